"""The cuts that the library chooses for the on-chip PCG (gbsimp_chip_plan, host only): within the kernel's
limits, with room in its lists for what each box of the cut holds, and where the chip's range ends."""
import ctypes as C
import itertools
import subprocess
import sys

import numpy as np
import pytest

from genpipeline_gb300 import _lib as L

NAMES = ("blocks", "Px", "Py", "Pz", "G", "NYm", "NZm", "stride", "q", "items", "multi", "terms", "smem")


def plan(grid, sms=152):
    v = (C.c_int32 * 13)()
    L.check(L.load().gbsimp_chip_plan(*grid, sms, v))
    return dict(zip(NAMES, v))


def axis_boxes(n, P):
    """(length, shared below, shared above) of the boxes of an axis, each kind once."""
    return {(n // P + (a < n % P), a > 0, a + 1 < P) for a in range(P)}


def grids():
    rng = np.random.default_rng(17)
    out = [(n, n, n) for n in (1, 2, 3, 8, 32, 57, 60, 64, 66)] + [(5000, 1, 1), (1, 1, 440), (1, 300, 300), (4, 4, 446)]
    while len(out) < 120:
        g = tuple(int(round(np.exp(rng.uniform(0, np.log(300))))) for _ in range(3))
        if np.prod(g) < 300_000:
            out.append(g)
    return out


@pytest.mark.parametrize("sms", [132, 148, 152])
def test_room_for_every_box(sms):
    held = 0
    for grid in grids():
        p = plan(grid, sms)
        if p["blocks"] == 0:
            continue
        held += 1
        cuts = (p["Px"], p["Py"], p["Pz"])
        assert p["blocks"] == np.prod(cuts) <= sms and all(P <= n for P, n in zip(cuts, grid))
        most = [-(-n // P) for n, P in zip(grid, cuts)]
        assert (p["NYm"], p["NZm"]) == (most[1] + 1, most[2] + 1)
        assert p["stride"] == np.prod([m + 1 for m in most]) and most[2] <= 32 and p["smem"] <= 227 * 1024
        G = p["G"]
        for kind in itertools.product(*(axis_boxes(n, P) for n, P in zip(grid, cuts))):
            (ex, ey, ez), lo, hi = zip(*kind)
            step = -(-ex // (2 * G))
            assert -(-ey // (32 // ez)) * G <= 8 and G * (step + 1) * p["NYm"] * p["NZm"] <= 256 * p["q"] <= 256 * 6
            # copies of each x plane: the last plane of a slab is also the first of the next
            copies = np.zeros(ex + 1, dtype=int)
            for i in (s * step + t for s in range(2 * G) for t in range(step + 1)):
                if i <= ex:
                    copies[i] += 1
            assert (copies >= 1).all()
            shared = []
            for n, below, above in kind:
                v = np.zeros(n + 1, dtype=int)
                v[0] |= below
                v[n] |= above
                shared.append(v)
            axes = shared[0][:, None, None] + shared[1][None, :, None] + shared[2][None, None, :]
            places = np.broadcast_to(copies[:, None, None], axes.shape)
            assert (places * (2 ** axes - 1)).sum() <= p["items"]
            assert places[axes > 1].sum() <= p["multi"] and (places * 2 ** axes)[axes > 1].sum() <= p["terms"]
            assert (axes > 0).sum() <= p["items"] and p["stride"] < 1 << 16 and p["terms"] < 1 << 16
    assert held > 60


def test_where_the_range_ends():
    for sms in (148, 152):
        assert plan((66, 66, 66), sms)["blocks"] > 0
        assert plan((67, 67, 67), sms)["blocks"] == 0
    assert plan((64, 64, 447))["blocks"] == 0  # rows longer than the modal form takes
    assert plan((192, 96, 96))["blocks"] == 0


def test_bad_arguments_are_refused():
    v = (C.c_int32 * 13)()
    lib = L.load()
    assert lib.gbsimp_chip_plan(0, 4, 4, 152, v) == L.GBS_EINVAL
    assert lib.gbsimp_chip_plan(4, 4, 4, 0, v) == L.GBS_EINVAL
    assert lib.gbsimp_chip_plan(4, 4, 4, 152, None) == L.GBS_EINVAL


def test_no_exception_leaves_the_library():
    """A search that finds no memory for its table says so; the process lives on."""
    code = (
        "import ctypes as C, resource\n"
        "lib = C.CDLL(%r)\n"
        "v = (C.c_int32 * 13)()\n"
        "size = int(open('/proc/self/statm').read().split()[0]) * resource.getpagesize()\n"
        "resource.setrlimit(resource.RLIMIT_AS, (size + 65536, size + 65536))\n"
        "print(lib.gbsimp_chip_plan(64, 64, 64, 152, v))\n" % L.library_path()
    )
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and int(r.stdout) in (L.GBS_OK, L.GBS_ENOMEM), (r.returncode, r.stderr[-500:])
