"""The single-matrix kernels on a system without unknowns: the column pointers'
only entries are written, and nothing else is read or written."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_factor_and_solve_without_unknowns(gpu, lib):
    import torch
    i32, f64 = torch.int32, torch.float64

    def dev(values, dtype):
        return torch.tensor(values, dtype=dtype, device="cuda")

    def p(t):
        return C.c_void_p(t.data_ptr())

    # The pointers hold what an earlier factorization left there.
    Lp, Up, Li, Ui = dev([3], i32), dev([3], i32), dev([2, 1, 0], i32), dev([2, 1, 0], i32)
    Lx, Ux = dev([1.0, 2.0, 3.0], f64), dev([1.0, 2.0, 3.0], f64)
    pinv, xi, cnt, x = dev([7, 7, 7], i32), torch.zeros(2048, dtype=i32, device="cuda"), dev([9, 9, 9], i32), dev([5.0], f64)
    Ap, Ai, Ax, q = dev([0], i32), dev([0], i32), dev([0.0], f64), dev([0], i32)
    c = cnt.data_ptr()
    assert lib.lusp_lu_factor_par_launch(0, p(Ap), p(Ai), p(Ax), p(q), p(Lp), p(Li), p(Lx), 3, p(Up), p(Ui), p(Ux), 3,
                                         p(pinv), p(xi), None, C.c_void_p(c), C.c_void_p(c + 4), C.c_void_p(c + 8),
                                         None) == 0
    torch.cuda.synchronize()
    assert cnt.tolist() == [0, 0, -1]
    assert Lp.tolist() == [0] and Up.tolist() == [0]
    assert Li.tolist() == [2, 1, 0] and Lx.tolist() == [1.0, 2.0, 3.0] and pinv.tolist() == [7, 7, 7]
    assert lib.lusp_trisolve_par_launch(0, p(Lp), p(Li), p(Lx), p(Up), p(Ui), p(Ux), p(pinv), p(q), p(Ax), p(x), p(xi),
                                        p(Lx), None) == 0
    torch.cuda.synchronize()
    assert x.tolist() == [5.0]
