"""The heat bath's warp-wide rejection loops and the two-lanes-per-site pass of the plugin level, at
the sizes and temperatures where they can go wrong: lattices below and above the size from which two
lanes per site are used, there with an odd number of 8-site tiles (the last warp half idle), timeslice
ranges that start and end inside a tile, long rejection loops (screened trials) and loops that run
into their bound.

Tolerances: the update depends on the coupling's direction, so the rounding of the eight-link sum
(a few 2^-52 of O(8)) is amplified by 8 / |a|; the fields have up to some ten thousand couplings, the
smallest about 1e-2 (1e-4 after MAG's cancellation), which bounds the difference of two FP64
evaluations by about 1e-10 per subgroup step; 1e-8 leaves room for six of them in a row.  The random rule multiplies by an element that does not depend on the
links: rounding of nine products, 1e-5 in FP32.
"""
import ctypes

import numpy as np
import pytest

import _oracle as O
from su3_ma_gauge_gpu_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def _rows(U, size):
    return U.reshape(4, 3, 3, 2, O.volume(size))[:, :2].astype(np.float64)


@pytest.mark.parametrize("gauge,size,T", [(O.LANDAU, (2, 2, 2, 6), 30.0), (O.MAG, (2, 2, 2, 6), 30.0),
                                          (O.U1XU1, (2, 4, 2, 6), 30.0), (O.COULOMB, (1, 2, 4, 6), 30.0),
                                          (O.LANDAU, (2, 2, 22, 110), 20.0), (O.MAG, (2, 2, 22, 110), 2.0),
                                          (O.U1XU1, (2, 2, 22, 110), 2.0), (O.COULOMB, (1, 22, 22, 20), 20.0)])
def test_long_rejection_loops_match_oracle(cuda, gauge, size, T):
    from su3_ma_gauge_gpu_b200 import _lib

    torch = cuda
    U = S.smooth_config(size, 0.3, 21)[0] if gauge != O.COULOMB else O.set_hot(size, 21, 1)
    D = O.set_hot(size, 22, 1) if gauge == O.COULOMB else None
    dU = torch.from_numpy(U.copy()).cuda()
    dD = torch.from_numpy(D.copy()).cuda() if D is not None else None
    for parity in (0, 1):
        _lib.check(_lib.lib().gf_sa_step(gauge, 1, dU.data_ptr(), dD.data_ptr() if dD is not None else None,
                                         _lib.size_arg(size), parity, ctypes.c_float(T), 3, 5 + parity, None), "sa")
        O.step(U, size, gauge, O.SA, parity, T, 3, 5 + parity, Udw=D)
    assert np.abs(_rows(dU.cpu().numpy(), size) - _rows(U, size)).max() < 1e-8
    if D is not None:
        assert np.abs(_rows(dD.cpu().numpy(), size) - _rows(D, size)).max() < 1e-8


@pytest.mark.parametrize("size", [(2, 2, 2, 6), (2, 2, 98, 98)])
@pytest.mark.parametrize("precision,eps", [("double", 1e-12), ("float", 1e-5)])
def test_exhausted_rejection_loops_stay_in_su3(cuda, precision, eps, size):
    """T / |a| ~ 1e6: no trial is accepted within the bound, every site takes the Haar limit."""
    from su3_ma_gauge_gpu_b200 import LandauKernelsSU3

    torch = cuda
    U = S.smooth_config(size, 0.3, 23, dtype=np.float64 if precision == "double" else np.float32)[0]
    dU = torch.from_numpy(U.copy()).cuda()
    k = LandauKernelsSU3(size, precision)
    for parity in (0, 1):
        k.saStep(0, 0, dU, None, parity, 1e7, 3, parity)
    G = _rows(dU.cpu().numpy(), size)
    assert np.isfinite(G).all() and np.abs(G - _rows(U, size)).max() > 0.1
    r = G[:, :, :, 0] + 1j * G[:, :, :, 1]
    for a in range(2):
        for b in range(2):
            dot = (r[:, a] * np.conj(r[:, b])).sum(axis=1)
            assert np.abs(dot - (a == b)).max() < eps


@pytest.mark.parametrize("algo,real,size", [(O.SA, 1, (4, 2, 6, 2)), (O.SA, 1, (4, 2, 50, 50)),
                                            (O.RANDOM, 0, (4, 2, 6, 2)), (O.RANDOM, 0, (4, 2, 98, 98))])
@pytest.mark.parametrize("slices", [(1, 3), (0, 1), (3, 4)])
def test_timeslice_range_matches_oracle(cuda, algo, real, size, slices):
    """An odd number of half tiles per timeslice: the runs start and end inside an 8-site tile."""
    from su3_ma_gauge_gpu_b200 import _lib

    torch = cuda
    U = S.smooth_config(size, 0.3, 25, dtype=np.float64 if real else np.float32)[0]
    dU = torch.from_numpy(U.copy()).cuda()
    for parity in (0, 1):
        _lib.check(_lib.lib().gf_step_slices_at(O.LANDAU, real, algo, dU.data_ptr(), _lib.size_arg(size), parity,
                                                ctypes.c_float(0.8), 3, parity, *slices, 24, None), "slices")
        O.step_slices(U, size, O.LANDAU, algo, parity, *slices, param=0.8, seed=3, counter=parity, rng_site_offset=24)
    assert np.abs(_rows(dU.cpu().numpy(), size) - _rows(U, size)).max() < (1e-8 if real else 1e-5)
