"""The Krylov solve in shared memory at the edges of its range (needs a B200).

Shapes on both sides of its size limit (256 values), ragged blocks, unequal
MPO widths, and Krylov spaces whose vectors do not all fit in the buffer.
The bound is the one the general path is held to: 25 Lanczos steps on vectors
of a few hundred values lose a few hundred roundings at most, 1e-11 of the
largest value leaves two decades.
"""
import ctypes as C

import numpy as np
import pytest

from yaqs_julia_b200 import _abi as A

pytestmark = pytest.mark.gpu


def _f(a):
    return np.asfortranarray(a, dtype=np.complex128).reshape(-1, order="F").view(np.float64)


@pytest.mark.parametrize("chil,D,chir,wl,wr", [(1, 2, 1, 1, 1), (2, 4, 1, 5, 1), (1, 2, 3, 1, 8), (7, 2, 9, 3, 5),
                                               (8, 4, 8, 5, 5), (11, 2, 11, 4, 4), (16, 2, 8, 3, 3), (13, 2, 10, 3, 3),
                                               (16, 2, 8, 1, 16), (4, 4, 4, 5, 5)])
def test_small_solve_matches_oracle(oracle, chil, D, chir, wl, wr):
    from yaqs_julia_b200 import _lib
    ctx = _lib.default_context()
    rng = np.random.default_rng(chil * 7 + chir + D + wl)

    def rand(*shape):
        return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)

    Lh, Rh = (E + E.transpose(2, 1, 0).conj() for E in (rand(chil, wl, chil), rand(chir, wr, chir)))
    W = rand(wl, D, D, wr)
    W = W + W.transpose(0, 2, 1, 3).conj()
    x = rand(chil, D, chir)
    out = np.zeros(2 * x.size)
    for kdim, ex in ((1, 0.0), (6, 0.0), (25, 0.0), (25, 1e-12)):
        mv = C.c_int32(0)
        ctx.check(ctx._lib.yaqs_batched_expm_site(ctx.handle, 1, chil, D, chir, wl, wr, A.dptr(_f(Lh)),
                                                  A.dptr(_f(Rh)), A.dptr(_f(W)), A.dptr(_f(x)), 0.02, kdim, 1e-10, ex,
                                                  A.dptr(out), C.byref(mv)))
        ref, mvo = oracle.expm_site(Lh, Rh, W, x, 0.02, kdim=kdim, exit_tol=ex)
        ref = ref.reshape(-1, order="F")
        assert mv.value == mvo
        assert np.abs(out.view(np.complex128) - ref).max() < 1e-11 * np.abs(ref).max()
