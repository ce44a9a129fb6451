"""The discrete adjoint's device memory: the gradient does not depend on what it held
before nor on work of another stream, and every block goes back to where it came from."""
import ctypes
import gc

import pytest
import torch

from mosscap_b200 import problems as P


def _gradient(p, vy, steps):
    from mosscap_b200.adjoint import EulerSteps, kh_initial_state
    v = vy.clone().requires_grad_(True)
    g = torch.tensor(p.gamma, dtype=torch.float64, device="cuda", requires_grad=True)
    q = EulerSteps.apply(kh_initial_state(v, g, p), g, p, steps, 4)
    J = 0.5 * (q[0] ** 2).sum()
    gv, gg = torch.autograd.grad(J, (v, g))
    return gv, float(gg)


@pytest.mark.gpu
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


def _allocator(held, fail_at=None):
    """An allocator of memory full of ones, which has none at call `fail_at`."""
    from mosscap_b200 import capi
    calls = []

    def alloc(user, n):
        calls.append(n)
        if len(calls) - 1 == fail_at:
            return None
        t = torch.full((n,), 255, dtype=torch.uint8, device="cuda")
        held[t.data_ptr()] = t
        return t.data_ptr()

    return capi.McAllocator(capi.ALLOC_FN(alloc), capi.FREE_FN(lambda user, p: held.pop(p, None) is None and 1 / 0),
                            None), calls


def _run(lib, p, mem, steps, every=4):
    """(status, gradient of the final density's sum) with the given memory."""
    from mosscap_b200 import capi
    from mosscap_b200.adjoint import _scheme, grid_of, pad_periodic
    grid, scheme, h = grid_of(p), _scheme(p, p.gamma), ctypes.c_void_p()
    st = lib.mc_adjoint_create_in(ctypes.byref(grid), ctypes.byref(scheme), every,
                                  ctypes.byref(mem) if mem else None, ctypes.byref(h))
    if st:
        assert not h.value
        return st, None
    q = pad_periodic(torch.tensor(p.Q[:, 0, p.ng:-p.ng, p.ng:-p.ng], device="cuda"), p.ng)
    lam = torch.zeros_like(q)
    lam[0, 0, p.ng:-p.ng, p.ng:-p.ng] = 1.0
    clk = capi.McClock(0.0, 1e300, 0.0, 1e300)
    stream, g = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.c_double()
    st = lib.mc_adjoint_forward(h, ctypes.c_void_p(q.data_ptr()), ctypes.byref(clk), steps, stream)
    if not st:
        st = lib.mc_adjoint_backward(h, ctypes.c_void_p(lam.data_ptr()), ctypes.byref(g), stream)
    assert lib.mc_adjoint_destroy(h) == 0
    return st, lam[:, 0, p.ng:-p.ng, p.ng:-p.ng].clone()


@pytest.mark.gpu
def test_callers_memory_with_any_contents_and_running_out(gpu_lib):
    p = P.kelvin_helmholtz_2d(32)
    st, want = _run(gpu_lib, p, None, 6)
    assert st == 0
    held = {}
    mem, calls = _allocator(held)
    st, got = _run(gpu_lib, p, mem, 6)
    assert st == 0 and torch.equal(got, want) and not held
    n = len(calls)
    assert n > 10
    for k in range(n):
        mem, calls = _allocator(held, k)
        st, _ = _run(gpu_lib, p, mem, 6)
        assert st != 0 and len(calls) == k + 1 and not held, k


@pytest.mark.gpu
def test_memory_goes_back(gpu_lib):
    """Nothing of a pass's memory stays out of torch's reach."""
    from mosscap_b200.adjoint import kh_vy
    p = P.kelvin_helmholtz_2d(400)
    small = P.kelvin_helmholtz_2d(16)
    _gradient(small, torch.tensor(kh_vy(small), device="cuda"), 8)  # kernels loaded
    vy = torch.tensor(kh_vy(p), device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    allocated, free = torch.cuda.memory_allocated(), torch.cuda.mem_get_info()[0]
    torch.cuda.reset_peak_memory_stats()
    _gradient(p, vy, 8)
    torch.cuda.synchronize()
    # the segment alone: 13 states of 4 variables
    assert torch.cuda.max_memory_allocated() - allocated > 13 * 4 * 8 * 406 * 406
    assert torch.cuda.memory_allocated() == allocated
    torch.cuda.empty_cache()
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20


@pytest.mark.gpu
@pytest.mark.parametrize("calls", [0, 3, 15])
def test_torch_running_out_of_memory_is_its_own_error(gpu_lib, monkeypatch, calls):
    """In mc_adjoint_create_in (0, 3) and in mc_adjoint_forward (15); the next pass works."""
    from mosscap_b200.adjoint import kh_vy
    p = P.kelvin_helmholtz_2d(16)
    vy = torch.tensor(kh_vy(p), device="cuda")
    want, _ = _gradient(p, vy, 5)
    real, left = torch.cuda.caching_allocator_alloc, [calls]

    def alloc(n):
        if left[0] == 0:
            raise torch.OutOfMemoryError("planned")
        left[0] -= 1
        return real(n)

    before = torch.cuda.memory_allocated()
    with monkeypatch.context() as m:
        m.setattr(torch.cuda, "caching_allocator_alloc", alloc)
        with pytest.raises(torch.OutOfMemoryError, match="planned"):
            _gradient(p, vy, 5)
    gc.collect()
    assert torch.cuda.memory_allocated() == before
    got, _ = _gradient(p, vy, 5)
    assert torch.equal(got, want)


def test_allocator_needs_both_functions():
    from mosscap_b200 import capi
    from mosscap_b200.adjoint import _scheme, grid_of
    lib = capi.load()
    p = P.kelvin_helmholtz_2d(16)
    grid, scheme, h = grid_of(p), _scheme(p, p.gamma), ctypes.c_void_p()
    mem = capi.McAllocator()
    assert lib.mc_adjoint_create_in(ctypes.byref(grid), ctypes.byref(scheme), 4, ctypes.byref(mem),
                                    ctypes.byref(h)) == 1
    assert not h.value
