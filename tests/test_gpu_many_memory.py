"""Calls on a GPU whose memory is nearly used up. energy_grad_many without the buffers with which several evaluations run at once
gives the same bits with one evaluation at a time; a Monte Carlo move that fails for memory can be made once there is some."""
import contextlib
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def nearly_full(gpu):
    """A context in which no piece of `left` bytes or more can be allocated on the GPU."""
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    try:
        cudart = ctypes.CDLL("libcudart.so.12")
    except OSError:
        pytest.skip("no CUDA runtime library to hold memory with")

    @contextlib.contextmanager
    def fill(left):
        torch.cuda.synchronize()
        held, size = [], 1 << 33
        while size >= left:
            at = ctypes.c_void_p()
            if cudart.cudaMalloc(ctypes.byref(at), ctypes.c_size_t(size)) == 0:
                held.append(at)
            else:
                size //= 2
        cudart.cudaGetLastError()
        try:
            yield
        finally:
            for at in held:
                cudart.cudaFree(at)
    return fill


def test_many_without_room_for_lanes(gpu, nearly_full):
    d, N, P = 3, 2000, 8
    basis = np.eye(d) * N ** (1.0 / d)
    modes, V = gpu.stealthy_kset(d, basis, N, 0.45)
    frac = np.random.default_rng(4).random((P, N, d))
    want = gpu.CCPotential(d, basis, modes, V)
    E0, F0 = want.energy_grad_many(frac)   # (and loads every kernel)
    p = gpu.CCPotential(d, basis, modes, V)
    p.energy_grad_many(np.random.default_rng(5).random((4, 2 * N, d)))   # the handle's buffers, for P configurations of N
    p.energy_grad_many(frac[:4])
    p.check_device_error()
    with nearly_full(1 << 20):   # a lane takes 5 MB
        E1, F1 = p.energy_grad_many(frac)
    assert np.array_equal(E1, E0) and np.array_equal(F1, F0)
    E2, F2 = p.energy_grad_many(frac)   # with room again
    assert np.array_equal(E2, E0) and np.array_equal(F2, F0)


def test_mc_move_after_one_without_memory(gpu, nearly_full):
    """The move's arrays (the modes, their weights, two copies of rho: 2.4 to 4.8 MB each) are not to be had."""
    g = np.stack(np.meshgrid(np.arange(1, 549), np.arange(-274, 274), indexing="ij"), -1).reshape(-1, 2)
    V = np.random.default_rng(2).random(len(g))
    x = np.random.default_rng(3).random((30, 2))
    new = np.array([0.3, 0.6])
    want = gpu.CCPotential(2, np.eye(2), g, V)
    want.set_configuration(x)
    dE = want.try_move(x[4], new)
    p = gpu.CCPotential(2, np.eye(2), g, V)
    p.set_configuration(x)
    p.energy()
    with nearly_full(1 << 20):
        with pytest.raises(gpu.CCError):
            p.try_move(x[4], new)
        with pytest.raises(gpu.CCError):
            p.try_move(x[4], new)
    assert p.try_move(x[4], new) == dE
