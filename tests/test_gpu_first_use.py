"""What a handle's first evaluations take: the arrays of the line plan are there from the first FP64 evaluation on, not from the
handle's creation (sets evaluated in mixed precision alone never need them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_handles_hold_no_line_arrays_before_fp64(gpu):
    torch = pytest.importorskip("torch")
    d, N, count = 2, 20000, 80
    basis = np.eye(d) * N ** (1.0 / d)
    modes, V = gpu.stealthy_kset(d, basis, N, 0.2)
    first = gpu.CCPotential(d, basis, modes, V)
    nslot = first.plan_info(N)["nseg"] * 8
    # slots: rho, u and a weight; modes: rho and a slot number; segments 20 bytes; tables and rounding a tenth
    expected = 1.1 * (nslot * 40 + len(V) * 20 + nslot // 8 * 20)
    torch.cuda.synchronize()

    def handles(m):
        before = torch.cuda.mem_get_info()[0]
        made = [gpu.CCPotential(d, basis, modes[:m], V[:m]) for _ in range(count)]
        return made, (before - torch.cuda.mem_get_info()[0]) / count

    used, _ = handles(1)        # (take up what earlier handles gave back)
    small, apart = handles(1)   # what a handle takes apart from its set (a stream)
    pots, each = handles(len(V))
    each -= apart
    print(f"{each:.0f} bytes a handle, expected {expected:.0f} (and up to 4 MB for all)")
    assert each <= expected + (4 << 20) / count
    # and the first FP64 evaluation of each is right
    frac = np.random.default_rng(1).random((500, d))
    first.set_configuration(frac)
    E = first.energy()
    for p in (pots[0], pots[-1]):
        p.set_configuration(frac)
        p.energy(gpu.PREC_MIXED)
        assert p.energy() == E
