"""The plan of the tcgen05 dC kernel, on the host: the partials that its CTAs write for a slab are the ones that are added
for it, and they fit the scratch."""
import ctypes
import random

import pytest

from sparsespline_ffn_b200 import _lib, build

# (N, h, L, r, spline_order): few keys and many tokens, where one run per SM is shorter than a slab
FEW_KEYS = [(94720, 32, 22, 128, 2), (258112, 64, 22, 128, 2), (513856, 256, 22, 32, 2), (897472, 512, 10, 16, 2),
            (1 << 21, 8, 22, 16, 2), (123456, 100, 22, 20, 2), (94720, 16, 21, 32, 1)]


def _plan(lib, p, slab=0):
    out = (ctypes.c_int64 * 8)()
    _lib.check(lib.skv_debug_dc_plan(ctypes.byref(p), slab, out))
    return dict(zip(("crosses", "tiles", "pitch", "run", "total", "slots", "keys", "added"), out))


def _check(lib, N, h, L, r, order):
    p = _lib.Problem(N=N, h=h, L=L, r=r, grid_lo=-3.0, scale=1.0, lambda_scale=1.0, activation=0, dtype=0, impl=2,
                     spline_order=order)
    if lib.skv_resolve_impl(ctypes.byref(p)) != _lib.SKV_IMPL["tcgen05"]:
        return False                                     # its operands do not fit shared memory
    d = _plan(lib, p)
    slabs = -(-h // d["keys"])
    assert d["total"] == slabs * d["pitch"] and d["pitch"] >= d["tiles"] == -(-N // 64)
    # walk the runs as the kernel does: a CTA of a plan that does not cross slabs works on one segment only
    written = [set() for _ in range(slabs)]
    covered = [0] * slabs
    for cta in range(-(-d["total"] // d["run"])):
        at, end = cta * d["run"], min(d["total"], (cta + 1) * d["run"])
        while at < end:
            slab, begin = divmod(at, d["pitch"])
            places = min(d["pitch"] - begin, end - at)
            tiles = min(d["tiles"] - begin, places)
            assert tiles >= 1, (N, h, L, r, order, d)
            slot = cta - slab * d["pitch"] // d["run"]
            assert slot not in written[slab]
            written[slab].add(slot)
            covered[slab] += tiles
            at += places
            if not d["crosses"]:
                assert at == end, (N, h, L, r, order, d)
    for slab in range(slabs):
        added = _plan(lib, p, slab)["added"]
        assert covered[slab] == d["tiles"]
        assert written[slab] == set(range(added)) and added <= d["slots"], (N, h, L, r, order, slab, d)
    return True


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.load()


@pytest.mark.parametrize("case", FEW_KEYS, ids=str)
def test_partials_written_are_the_ones_added(lib, case):
    assert _check(lib, *case)


def test_partials_over_the_range_of_shapes(lib):
    rng = random.Random(3)
    checked = 0
    for _ in range(400):
        order = rng.choice([1, 2, 2, 2])
        N = int(2 ** rng.uniform(0, 21)) if rng.random() < 0.5 else 64 * int(2 ** rng.uniform(0, 15))
        checked += _check(lib, N, int(2 ** rng.uniform(0, 12.5)), rng.randint(4, 64),
                          rng.choice([1, 16, 20, 32, 64, 96, 128]), order)
    assert checked > 200


def test_token_and_place_counts_stay_within_32_bits(lib):
    def problem(N, h, r=16, impl=0):
        return _lib.Problem(N=N, h=h, L=22, r=r, grid_lo=-3.0, scale=1.0, lambda_scale=1.0, activation=0, dtype=0, impl=impl)

    def resolve(*a, **k):
        return lib.skv_resolve_impl(ctypes.byref(problem(*a, **k)))

    # dz addresses a tile's rows by a 32-bit coordinate: beyond it, the CUDA-core kernels
    last = 2**31 - 257
    assert resolve(last, 8) == _lib.SKV_IMPL["tcgen05"]
    for N in (last + 1, 2**31, 2**32, 2**40):
        assert resolve(N, 8) == _lib.SKV_IMPL["simt"] and resolve(N, 8, impl=2) == -3
        for op in (_lib.SKV_OP_FORWARD, _lib.SKV_OP_BACKWARD):
            assert lib.skv_scratch_bytes(ctypes.byref(problem(N, 8)), op) < 2**63
    # dC counts 64-token tiles of all slabs in 32 bits
    for N, h in ((last, 5120), (2**30, 1 << 20), (2**28, 1 << 24)):
        if resolve(N, h, r=128) == _lib.SKV_IMPL["tcgen05"]:
            d = _plan(lib, problem(N, h, r=128))
            assert d["total"] == -(-h // d["keys"]) * d["pitch"] < 2**31 and d["tiles"] <= d["pitch"]
