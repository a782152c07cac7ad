"""The plugin steps of lattices that run with two lanes per site (just above that size, an odd number of
8-site tiles, so the last warp is half idle) against the same step taken timeslice by timeslice, whose
smaller ranges run with four lanes per site and start inside a tile: bit for bit, because the sites of one
parity share no link and both layouts do the same arithmetic (MAG's SR in FP64: two evaluations that differ by
rounding, whatever the layout of the whole pass).  Coulomb slices, which have no timeslice
ranges, against the FP64 oracle: two FP64 evaluations of a coupling |a| > 1e-3 differ by about
8 / |a| x 2^-52 per subgroup step, well below 1e-8 for six steps."""
import ctypes

import numpy as np
import pytest

import _oracle as O
from su3_ma_gauge_gpu_b200 import synthetic as S

pytestmark = pytest.mark.gpu

PARAM = {O.OR: 1.7, O.SA: 0.8, O.SR: 0.5}


def _step(L, gauge, real, algo, dU, dD, size, parity):
    s = (ctypes.c_int32 * 4)(*size)
    p = ctypes.c_float(PARAM.get(algo, 0.0))
    a = (gauge, real, dU.data_ptr(), dD.data_ptr() if dD is not None else None, s, parity)
    if algo == O.OR:
        return L.gf_or_step(*a, p, None)
    if algo == O.MICRO:
        return L.gf_micro_step(*a, None)
    if algo == O.RANDOM:
        return L.gf_random_trafo(*a, 3, parity, None)
    return (L.gf_sa_step if algo == O.SA else L.gf_sr_step)(*a, p, 3, parity, None)


@pytest.mark.parametrize("real,size", [(0, (2, 2, 98, 98)), (1, (2, 2, 138, 138))], ids=["fp32", "fp64"])
@pytest.mark.parametrize("gauge", [O.LANDAU, O.MAG, O.U1XU1], ids=["landau", "mag", "u1xu1"])
def test_whole_pass_equals_timeslice_passes(cuda, gauge, real, size):
    from su3_ma_gauge_gpu_b200 import _lib

    torch = cuda
    L = _lib.lib()
    U = torch.from_numpy(S.smooth_config(size, 0.3, 61, dtype=np.float64 if real else np.float32)[0]).cuda()
    for algo in (O.OR, O.MICRO, O.SA, O.SR, O.RANDOM):
        A, B = U.clone(), U.clone()
        for parity in (0, 1):
            _lib.check(_step(L, gauge, real, algo, A, None, size, parity), "step")
            for t in range(size[0]):
                _lib.check(L.gf_step_slices(gauge, real, algo, B.data_ptr(), _lib.size_arg(size), parity,
                                            ctypes.c_float(PARAM.get(algo, 0.0)), 3, parity, t, t + 1, None), "slices")
        if (gauge, real, algo) == (O.MAG, 1, O.SR):
            # the compiler contracts this rule differently in the range pass; two FP64 evaluations
            assert (A - B).abs().max().item() < 1e-8
        else:
            assert torch.equal(A, B), algo
        assert not torch.equal(A, U)


@pytest.mark.parametrize("algo", [O.OR, O.MICRO, O.SR, O.RANDOM], ids=["or", "micro", "sr", "random"])
def test_coulomb_slice_matches_oracle(cuda, algo):
    from su3_ma_gauge_gpu_b200 import _lib

    torch = cuda
    size = (1, 42, 42, 44)
    U, D = O.set_hot(size, 3, 1), O.set_hot(size, 4, 1)
    dU, dD = torch.from_numpy(U.copy()).cuda(), torch.from_numpy(D.copy()).cuda()
    for parity in (0, 1):
        _lib.check(_step(_lib.lib(), O.COULOMB, 1, algo, dU, dD, size, parity), "step")
        O.step(U, size, O.COULOMB, algo, parity, PARAM.get(algo, 0.0), 3, parity, Udw=D)
    V = O.volume(size)
    for got, want in ((dU, U), (dD, D)):
        rows = [np.asarray(x).reshape(4, 3, 3, 2, V)[:, :2] for x in (got.cpu().numpy(), want)]
        assert np.abs(rows[0] - rows[1]).max() < 1e-8
