"""The kernels that the benchmark's roofline names."""
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


def test_largest_kernel_is_named_whether_or_not_its_bytes_are_known():
    import bench
    prof = {"sweep_zeta": [1.5, 9], "weno_faces": [1.7, 18], "sweep_xi": [1.1, 9], "prim_ghost_fill": [0.6, 18]}
    assert bench.largest_kernels(prof) == ("weno_faces", "sweep_zeta")
    assert bench.largest_kernels({**prof, "weno_faces": [0.2, 18]}) == ("sweep_zeta", "sweep_zeta")
