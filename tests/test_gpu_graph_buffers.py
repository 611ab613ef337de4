"""A program's own CUDA graphs of evaluations keep their buffers: an evaluation of the same handle and particle count in the
other precision, rho and S(k) in between allocate, but never move what the graph reads and writes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["mixed", "fp64"])
@pytest.mark.parametrize("d,N,chi", [(2, 2000, 0.2), (3, 2000, 0.45)])
def test_graph_survives_the_other_precision(gpu, d, N, chi, first):
    torch = pytest.importorskip("torch")
    basis = np.eye(d) * N ** (1.0 / d)
    modes, V = gpu.stealthy_kset(d, basis, N, chi)
    p = gpu.CCPotential(d, basis, modes, V)
    p.set_path(gpu.PATH_SPLIT)
    start = np.random.default_rng(3).random((N, d))
    frac = torch.from_numpy(start).cuda()
    E = torch.zeros(1, dtype=torch.float64, device="cuda")
    F = torch.zeros(N, d, dtype=torch.float64, device="cuda")
    prec, other = (gpu.PREC_MIXED, gpu.PREC_FP64) if first == "mixed" else (gpu.PREC_FP64, gpu.PREC_MIXED)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def evaluate(precision):
        p.energy_grad_device(N, frac.data_ptr(), E.data_ptr(), F.data_ptr(), precision=precision,
                             stream=stream.cuda_stream)

    evaluate(prec)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        evaluate(prec)
    graph.replay()
    torch.cuda.synchronize()
    E0, F0 = E.clone(), F.clone()
    evaluate(other)
    stream.synchronize()
    p.set_configuration(start)
    p.rho()
    p.structure_factor(modes)
    # whatever was given back to the driver now holds NaN
    fill = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for n in [1 << k for k in range(10, 22)] * 4]
    torch.cuda.synchronize()
    E.zero_()
    F.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(E, E0) and torch.equal(F, F0)
    assert all(bool(torch.isnan(x).all()) for x in fill)   # and it wrote into none of it
