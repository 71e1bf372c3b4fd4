"""Shared helpers of the test suite."""
import numpy as np

# (group, (Lx, Ly, Lz, Lt), ndims): SU(2) in d = 2, 3, 4 and U(1) in d = 2, 4
GEOMS = [
    (0, (4, 4, 4, 4), 4),
    (0, (4, 2, 2, 6), 4),
    (0, (6, 1, 1, 4), 2),
    (0, (4, 6, 1, 4), 3),
    (1, (4, 4, 4, 4), 4),
    (1, (8, 1, 1, 6), 2),
]
GEOM_IDS = [f"{'su2' if g == 0 else 'u1'}-{'x'.join(map(str, d))}-d{nd}" for g, d, nd in GEOMS]


def rel(a, b):
    """Norm-wise relative difference |a - b| / |b|."""
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def group_name(g):
    return "su2" if g == 0 else "u1"


def context_setting(lattice, what, value):
    """A setting of the lattice's context that only tests use (su2b_ctx.h)."""
    import ctypes as C
    f = lattice.lib.su2b_test_set
    f.argtypes, f.restype = [C.c_void_p, C.c_int, C.c_long], C.c_int
    assert f(lattice.ctx, what, value) == 0


def fail_allocations(lattice, n):
    """The next n device allocations of the lattice's context ask for more than a device has."""
    context_setting(lattice, 0, n)


def leave_error(lattice):
    """An error of this thread's CUDA runtime that nobody has looked at."""
    context_setting(lattice, 2, 0)


def wait_limit(lattice, n):
    """The polls or cycles after which a wait of the tiled solves gives up (-1: their own)."""
    context_setting(lattice, 1, n)
