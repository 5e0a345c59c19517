// softfp_harness.cpp with the estimates moved by a part of their error bounds
// (argv[3]: -1 to 1) instead of units in the last place.
#define main patterns
#include "softfp_harness.cpp"
#undef main

int main(int argc, char** argv) {
  sf::est_relative() = atof(argv[3]);
  char zero[] = "0";
  char* args[] = {argv[0], argv[1], argv[2], zero};
  return patterns(4, args);
}
