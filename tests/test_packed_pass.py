"""The packed two-links-at-a-time FP32 pass (launch shape 7 of contexts without the separate W array)
against the direct pass, bit for bit: both take the products and sums in the same order.  Sizes: an odd
number of 8-site tiles (half a warp idle), a batch of uneven lattices, a lattice of several tiles per
persistent warp; Coulomb slices, whose temporal planes hold W and have no down link."""
import pytest

from su3_ma_gauge_gpu_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capped", [False, True], ids=["plain", "capped"])
@pytest.mark.parametrize("sizes", [[(2, 2, 2, 6)], [(4, 6, 10, 8), (2, 2, 2, 6), (6, 4, 4, 8)], [(16, 16, 16, 16)]],
                         ids=["odd_tiles", "batch", "many_tiles"])
@pytest.mark.parametrize("gauge", ["landau", "mag", "u1xu1", "coulomb"])
def test_packed_pass_bit_identical_to_direct(cuda, gauge, sizes, capped):
    from su3_ma_gauge_gpu_b200.engine import GaugeFixer

    torch = cuda
    if gauge == "coulomb":
        sizes = [(s[0],) + ((2, 4, 6) if s[1] * s[2] * s[3] % 16 else s[1:]) for s in sizes]
    fields = []
    for k, s in enumerate(sizes):
        U = S.smooth_config(s, 0.3, 41 + k)[0]
        fields.append(torch.from_numpy(S.gpupattern_to_timeslices(U, s) if gauge == "coulomb" else U).cuda())
    results = []
    for variant in (0, 7):
        with GaugeFixer(sizes, gauge=gauge, mixed="refine" if gauge == "coulomb" else True) as gf:
            gf.set_pass_shape("fp32", variant)
            if variant == 7:
                gf.set_pass_order("fp32", True, capped)
            for k, f in enumerate(fields):
                gf.load(k, f)
            gf.sweeps("or", 3, 1.7)
            gf.sweeps("micro", 2)
            outs = [torch.empty_like(f) for f in fields]
            for k, o in enumerate(outs):
                gf.store(k, o)
            results.append(outs)
    for a, b, f in zip(*results, fields):
        assert torch.equal(a, b)
        assert not torch.equal(a, f)
