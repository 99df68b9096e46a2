"""What the host side of the library does when the runtime refuses something, and in which order it
prepares memory: the library's objects linked with a stand-in for the CUDA runtime
(fake_cudart.cpp), so no GPU is needed and no kernel runs."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

from flame3d_mhd_gb300 import abi
from flame3d_mhd_gb300 import build as b

HERE = Path(__file__).resolve().parent
PER = [dict(kind=abi.BC_PERIODIC)] * 6
OUT_OF_MEMORY, INVALID = 2, 1  # cudaErrorMemoryAllocation, cudaErrorInvalidValue


class Host:
    """One context on the stand-in runtime; arrays are addresses that nothing reads."""

    def __init__(self, lib, **kw):
        self.lib, self.P = lib, abi.make_params(20, 12, 8, bc=PER, **{"viscous": 0, **kw})
        lib.fake_reset()
        self.ctx = C.c_void_p()
        self.array = (C.c_void_p(0x500000000000 + (k << 24)) for k in range(1 << 20))
        self.plane = 28 * 20 * 16

    def create(self, ok=True):
        rc = self.lib.f3d_create(C.byref(self.P), C.byref(self.ctx))
        assert (rc == 0) == ok
        return self

    def metrics(self, stream=0x77):
        m = (C.c_void_p * 9)(*[next(self.array) for _ in range(9)])
        assert self.lib.f3d_set_metrics(self.ctx, m, next(self.array), C.c_void_p(stream)) == 0
        return self

    def rhs(self, stream=0x77):
        return self.lib.f3d_rhs(self.ctx, next(self.array), next(self.array), C.c_void_p(stream))

    def vjp(self, stream=0x77):
        a = [next(self.array) for _ in range(3)]
        return self.lib.f3d_rhs_vjp(self.ctx, *a, C.c_void_p(stream))

    def log(self):
        """[(what, address, bytes, stream), ...] since the last call"""
        text = self.lib.fake_log().decode()
        new, self.seen = text[getattr(self, "seen", 0):], len(text)
        rows = [r.split() for r in new.splitlines()]
        return [(r[0], int(r[1], 16), int(r[2]), int(r[3], 16)) for r in rows]

    def close(self):
        if self.ctx:
            assert self.lib.f3d_destroy(self.ctx) == 0
            self.ctx = C.c_void_p()


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    b.build()
    d = tmp_path_factory.mktemp("fake")
    inc = Path(b.nvcc()).resolve().parent.parent / "include"
    so = d / "libhost.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{inc}", "-o", str(so),
                    str(HERE / "fake_cudart.cpp"), *map(str, sorted(b.BUILD.glob("*.o")))], check=True)
    lib = C.CDLL(str(so))
    real = abi.load()
    for name in abi.EXPORTED:
        getattr(lib, name).restype, getattr(lib, name).argtypes = getattr(real, name).restype, getattr(real, name).argtypes
    lib.fake_log.restype = C.c_char_p
    lib.fake_limit.argtypes, lib.fake_held.restype = [C.c_size_t], C.c_size_t
    lib.fake_refuse.argtypes = [C.c_char_p, C.c_int]
    yield lib
    lib.fake_reset()


@pytest.fixture
def host(lib):
    made = []

    def make(**kw):
        made.append(Host(lib, **kw))
        return made[-1]
    yield make
    lib.fake_reset()
    for h in made:
        h.close()


def _launches(rows, name):
    return [r for r in rows if r[0].startswith("launch:") and name in r[0]]


@pytest.mark.parametrize("first", ["metrics", "check", "filter"])
def test_memory_is_cleared_before_any_stream_uses_it(host, first):
    """Streams that do not wait for the legacy stream (PyTorch's pool streams) may be the first to use a
    context: what must be zero is cleared on the stream of the first call that needs it, once, and the
    adjoint's scratch, which the first reverse call takes, on that call's."""
    h = host(filter=abi.FILTER_NONLINEAR if first == "filter" else abi.FILTER_NONE).create()
    rows = h.log()
    held = [r for r in rows if r[0] == "malloc"]
    assert not any(r[0] == "memset" for r in rows)
    if first == "check":
        h.lib.f3d_check_finite(h.ctx, next(h.array), C.c_void_p(0x55))
    elif first == "filter":
        h.lib.f3d_filter(h.ctx, *[next(h.array) for _ in range(3)], C.c_void_p(0x55))
    else:
        h.metrics(0x55)
    rows = [r for r in h.log() if r[0] == "memset" and any(m[1] <= r[1] < m[1] + m[2] for m in held)]
    sizes = {r[2] for r in rows}
    assert 32 in sizes and any(s >= 8 * h.plane for s in sizes) and all(r[3] == 0x55 for r in rows)
    assert first != "filter" or 16 * h.plane in sizes
    h.metrics(0x66)
    assert not any(r[0] == "memset" for r in h.log())
    if first == "filter":
        return  # the adjoint has no filters
    h.metrics().log()
    assert h.vjp(0x99) == 0
    rows = h.log()
    taken = [r for r in rows if r[0] == "malloc"]
    assert len(taken) == 1
    sets = [r for r in rows if r[0] == "memset" and taken[0][1] <= r[1] < taken[0][1] + taken[0][2]]
    assert any(r[2] == taken[0][2] for r in sets) and all(r[3] == 0x99 for r in sets)


def test_a_refused_list_stops_the_right_hand_side(host):
    """Without its lists the WENO fluxes would be the previous state's."""
    h = host().create().metrics()
    h.log()
    h.lib.fake_refuse(b"k_weno_list", INVALID)
    assert h.rhs() == abi.F3D_ERR_CUDA
    rows = h.log()
    assert any(r[0].startswith("refused:") for r in rows)
    assert not _launches(rows, "k_weno_faces") and not _launches(rows, "k_sweep")
    h.lib.fake_reset()
    h.seen = 0
    assert h.rhs() == abi.F3D_OK


def test_lists_start_from_zero_after_a_refused_launch(host):
    """The counts of a listing whose later kernels were refused are cleared before the next one: lists
    appended behind them would run out of their arrays."""
    h = host().create().metrics()
    for call, refused in ((h.rhs, b"k_weno_faces"), (h.vjp, b"k_weno_vjp"), (h.vjp, b"k_sweep_vjp")):
        h.lib.fake_refuse(refused, INVALID)
        assert call() == abi.F3D_ERR_CUDA
        h.lib.fake_refuse(b"", 0)
        h.log()
        assert h.rhs() == abi.F3D_OK and h.vjp() == abi.F3D_OK
        clean, lists = set(), 0
        for what, at, size, _ in h.log():
            if what == "clears":
                clean.add(at)
            elif what == "memset":
                clean |= {at + k for k in range(0, size, 8)}
            elif what == "counts":
                assert at in clean, hex(at)
                clean.discard(at)  # the listing that follows uses them
                lists += 1
        assert lists == 2


def test_split_cotangents_start_from_zero_after_a_refused_launch(host):
    """The reverse sweeps clear the split-flux cotangents they read; where one of them was refused, the next
    reverse call clears them all first (and only then)."""
    h = host().create().metrics()
    planes = 30 * h.plane * 8
    cleared = lambda: sum(r[0] == "memset" and r[2] == planes for r in h.log())  # noqa: E731
    assert h.vjp() == abi.F3D_OK and cleared() == 0
    assert h.vjp() == abi.F3D_OK and cleared() == 0
    for refused in (b"k_weno_vjp", b"k_sweep_vjp"):
        h.lib.fake_refuse(refused, INVALID)
        assert h.vjp() == abi.F3D_ERR_CUDA
        h.lib.fake_refuse(b"", 0)
        h.log()
        assert h.vjp() == abi.F3D_OK and cleared() == 1
        assert h.vjp() == abi.F3D_OK and cleared() == 0


@pytest.mark.parametrize("viscous", [0, 1])
def test_reverse_without_room_for_the_listed_faces(host, viscous):
    """Where the device has room for the adjoint's scratch, but not for the split-flux cotangents of listed WENO
    faces beside it, the reverse runs with its WENO faces in the tiles; with less it is refused, and runs
    once there is room."""
    h = host(viscous=viscous)
    h.create().metrics()
    need = 8 * (h.plane * (6 + 25 + 24) + (24 * 16 * 12 * 24 if viscous else 0))
    spare = 64 * 1024  # rounding of the arrays
    h.lib.fake_limit(h.lib.fake_held() + need // 2)
    assert h.vjp() == abi.F3D_ERR_CUDA
    assert h.rhs() == abi.F3D_OK  # the refusal is not reported again
    h.lib.fake_limit(h.lib.fake_held() + need + spare)
    h.log()
    assert h.vjp() == abi.F3D_OK
    rows = h.log()
    assert not _launches(rows, "k_weno_vjp")
    assert len([r for r in _launches(rows, "k_sweep_vjp") if "ELi1EE" in r[0]]) == 3  # characteristic faces in the tiles
    assert h.vjp() == abi.F3D_OK


def test_right_hand_side_without_room_for_the_lists(host):
    """A context whose lists do not fit keeps its WENO faces in the tiles."""
    h = host().create()
    full = h.lib.fake_held()
    h.close()
    h.lib.fake_limit(full - 1)
    h.create().metrics().log()
    assert h.lib.fake_held() < full - 100 * h.plane
    h.lib.fake_limit(1 << 40)
    assert h.rhs() == abi.F3D_OK and h.vjp() == abi.F3D_OK
    rows = h.log()
    assert not _launches(rows, "k_weno")
    assert len([r for r in _launches(rows, "k_sweepIL") if "ELi1EdE" in r[0]]) == 3
