"""energy_grad_many on a GPU whose memory is nearly used up: the buffers with which several evaluations run at once are not to
be had, and the call gives the same bits with one evaluation at a time."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_many_without_room_for_lanes(gpu):
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    try:
        cudart = ctypes.CDLL("libcudart.so.12")
    except OSError:
        pytest.skip("no CUDA runtime library to hold memory with")
    d, N, P = 3, 2000, 8
    basis = np.eye(d) * N ** (1.0 / d)
    modes, V = gpu.stealthy_kset(d, basis, N, 0.45)
    frac = np.random.default_rng(4).random((P, N, d))
    want = gpu.CCPotential(d, basis, modes, V)
    E0, F0 = want.energy_grad_many(frac)   # (and loads every kernel)
    p = gpu.CCPotential(d, basis, modes, V)
    p.energy_grad_many(np.random.default_rng(5).random((4, 2 * N, d)))   # the handle's buffers, for P configurations of N
    p.energy_grad_many(frac[:4])
    torch.cuda.synchronize()
    held, size = [], 1 << 33
    while size >= 1 << 20:   # a lane takes 5 MB: leave less than 1 MB
        at = ctypes.c_void_p()
        if cudart.cudaMalloc(ctypes.byref(at), ctypes.c_size_t(size)) == 0:
            held.append(at)
        else:
            size //= 2
    cudart.cudaGetLastError()
    try:
        E1, F1 = p.energy_grad_many(frac)
    finally:
        for at in held:
            cudart.cudaFree(at)
    assert np.array_equal(E1, E0) and np.array_equal(F1, F0)
    E2, F2 = p.energy_grad_many(frac)   # with room again
    assert np.array_equal(E2, E0) and np.array_equal(F2, F0)
