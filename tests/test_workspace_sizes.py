"""CPU test of the workspace sizes: regions that held a call before digit products and unpadded channel rows are
still taken, and a chunk's buffers stay within the budget of 6 GiB (plus the FP64 tangents' 512 MiB)."""
import ctypes

import pytest

from deeperwin_gb300 import _lib


def _sizes(n, nu, N, K, B, prec, mode):
    L = _lib.lib()
    a = _lib.DwArch(n, nu, N, K, 1, 8, 256, 32, 32, 64, 64)
    return (L.dw_workspace_bytes(ctypes.byref(a), prec, B, mode), L.dw_debug_workspace_least_bytes(ctypes.byref(a), prec, B, mode))


# electrons, spin-up, ions, determinants, walkers, precision form, mode: bytes asked for before those changes
EARLIER = [
    (4, 2, 2, 8, 1, 3, 0, 640768),
    (4, 2, 2, 8, 1, 3, 1, 1188868),
    (4, 2, 2, 8, 2048, 3, 2, 229514240),
    (16, 8, 6, 32, 1, 1, 1, 16147984),
    (16, 8, 6, 32, 64, 3, 1, 933836288),
    (16, 8, 6, 32, 4096, 3, 1, 6440006144),
    (40, 20, 12, 64, 8, 3, 1, 1986060320),
    (40, 20, 12, 64, 1, 1, 1, 251019024),
    (20, 5, 12, 11, 2610, 1, 1, 6434561568),
    (51, 25, 10, 16, 336, 4, 1, 6271229504),
    (34, 24, 15, 8, 2723, 0, 1, 6405480332),
    (27, 14, 5, 8, 33, 4, 1, 834879876),
]


@pytest.mark.parametrize("case", EARLIER)
def test_earlier_workspaces_are_taken(case):
    full, least = _sizes(*case[:-1])
    assert least <= case[-1] and least <= full


@pytest.mark.parametrize("prec", range(6))
@pytest.mark.parametrize("shape", [(2, 1, 1, 4), (10, 5, 10, 16), (16, 8, 6, 32), (27, 14, 5, 8), (40, 20, 12, 64), (64, 32, 16, 128)])
def test_workspaces_stay_within_the_budget(prec, shape):
    for B in (1, 64, 4096, 100000):
        for mode in (0, 1, 2):
            full, least = _sizes(*shape, B, prec, mode)
            one = _sizes(*shape, 1, prec, mode)[0]
            # at least one walker; outputs and proposals of the walkers themselves; one geometry's maps
            assert 0 < least <= full <= max(one, (6 << 30) + (513 << 20)) + B * (4 * shape[0] * 16 + 1024)
