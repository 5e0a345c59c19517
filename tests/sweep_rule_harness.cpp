// C entry points over sweep_rule.h for the CPU tests.
#include "sweep_rule.h"

extern "C" {
long long choice(int variant, long long above) { return geon::sweep_choice(variant, above); }
int chosen(long long c, long long n) { return geon::sweep_variant(c, n); }
int kernel(int variant, long long n, int sms, int resident) { return geon::sweep_kernel(variant, n, sms, resident != 0); }
int ordered(long long n, int sms) { return geon::sweep_ordered(n, sms); }
long long tuned(const double* rates, long long n, int sms) { return geon::sweep_tuned(rates, n, sms); }
}
