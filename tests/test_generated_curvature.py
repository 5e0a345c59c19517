"""curvature_sparse.cuh is exactly what its generator writes (no hand edits)."""
import importlib.util
import os

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "geon_gb300", "csrc")


def test_sparse_curvature_header_is_generated():
    spec = importlib.util.spec_from_file_location("gen_sparse_christoffel", os.path.join(CSRC, "gen_sparse_christoffel.py"))
    gen = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(gen)
    with open(os.path.join(CSRC, "curvature_sparse.cuh")) as f:
        assert f.read() == gen.curvature_text()
