"""The discrete adjoint does not depend on what its device memory held before, nor on
work of another stream."""
import pytest
import torch

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu


def _gradient(p, vy, steps):
    from mosscap_b200.adjoint import EulerSteps, kh_initial_state
    v = vy.clone().requires_grad_(True)
    g = torch.tensor(p.gamma, dtype=torch.float64, device="cuda", requires_grad=True)
    q = EulerSteps.apply(kh_initial_state(v, g, p), g, p, steps, 4)
    J = 0.5 * (q[0] ** 2).sum()
    gv, gg = torch.autograd.grad(J, (v, g))
    return gv, float(gg)


def test_gradient_on_a_side_stream_beside_a_busy_default_stream(gpu_lib):
    """9, 20 and 9 steps: the memory of the records of the first run (9 + 1 doubles, the size
    of a control block) can serve the last one's control blocks, and the default stream
    does not run anything before the last run is over."""
    from mosscap_b200.adjoint import kh_vy
    p = P.kelvin_helmholtz_2d(48)
    vy = torch.tensor(kh_vy(p), device="cuda")
    want, want_gamma = _gradient(p, vy, 9)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for steps in (9, 20, 9):
        torch.cuda.synchronize()
        torch.cuda._sleep(1_000_000_000)  # about half a second of the default stream
        with torch.cuda.stream(side):
            got, got_gamma = _gradient(p, vy, steps)
        side.synchronize()
    assert torch.equal(got, want)
    assert got_gamma == want_gamma
    torch.cuda.synchronize()
