"""The operators under torch's tracing, transforms, threads and saved-tensor hooks."""
import math
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(seed, H=4, N=330, d=64):       # long enough for the tensor-core kernels of a mix
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(1, H, N, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    theta = torch.zeros(H, 3, 5, device="cuda")
    theta[:, 2, 2] = 1.0
    theta += 0.1 * torch.randn(H, 3, 5, device="cuda", generator=g)
    w = torch.eye(H, device="cuda") + 0.1 * torch.randn(H, H, device="cuda", generator=g)
    return q, k, v, theta, w


def _ops():
    import fmta_b200 as F
    scale = 1.0 / math.sqrt(64)
    return {
        "conv": lambda q, k, v, t, w: F.FlashConvAttentionCUDAFunction.apply(q, k, v, t, scale, 2, 2, True),
        "mix": lambda q, k, v, t, w: F.head_conv_attention(q, k, v, w, True, scale),
        "conv_mix": lambda q, k, v, t, w: F.conv_headmix_attention(q, k, v, t, w[None], True, scale),
    }


@pytest.mark.parametrize("name", ["conv", "mix", "conv_mix"])
@pytest.mark.parametrize("grad", [False, True])
def test_a_trace_computes(name, grad):
    """A traced operator answers new inputs, and differentiates, as the operator itself does."""
    op = _ops()[name]
    first, second = _inputs(0), _inputs(1)
    for t in first:
        t.requires_grad_(grad)
    traced = torch.jit.trace(op, first, check_trace=False)
    for t in second:
        t.requires_grad_(grad)
    got, want = traced(*second), op(*second)
    assert torch.equal(got, want)
    if grad:
        wrt = [t for t, used in zip(second, (1, 1, 1, name != "mix", name != "conv")) if used]
        do = torch.randn_like(want)
        for a, b in zip(torch.autograd.grad(got, wrt, do), torch.autograd.grad(want, wrt, do)):
            assert float((a.float() - b.float()).norm()) <= 4e-3 * float(b.float().norm())     # gradients rounded to bf16 on their own


@pytest.mark.parametrize("name", ["conv", "mix", "conv_mix"])
def test_compiled_around(name):
    op = _ops()[name]
    args = _inputs(2)
    torch._dynamo.reset()
    f = torch.compile(lambda *a: op(*a) * 2, backend="eager")
    assert torch.equal(f(*args), op(*args) * 2)


@pytest.mark.parametrize("name", ["conv", "mix", "conv_mix"])
@pytest.mark.parametrize("which", [0, 2, 3, 4])
@pytest.mark.parametrize("grad,grad_mode", [(False, True), (False, False), (True, True), (True, False)])
def test_forward_mode_is_refused(name, which, grad, grad_mode):
    """No tangent is dropped silently, whether or not the autograd node is passed by."""
    if (name, which) in (("conv", 4), ("mix", 3)):
        pytest.skip("not an input of the operator")
    op = _ops()[name]
    with torch.autograd.forward_ad.dual_level():
        args = [t.clone().requires_grad_(grad) for t in _inputs(3)]
        args[which] = torch.autograd.forward_ad.make_dual(args[which], torch.ones_like(args[which]))
        with torch.set_grad_enabled(grad_mode), pytest.raises((RuntimeError, NotImplementedError)):
            op(*args)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("conv", [False, True])
def test_backward_of_an_output_on_any_address(dtype, conv):
    """The output that the caller hands back may be a view that starts anywhere in a buffer."""
    import fmta_b200 as F
    q, k, v, theta, w = _inputs(4, N=300)
    th = theta if conv else None
    o, l, m, lse = F.conv_headmix_forward(q, k, v, w, th, 0.125, True, out_dtype=dtype)
    do = torch.randn(q.shape, device="cuda").to(torch.bfloat16)
    buf = torch.zeros(o.numel() + 8, dtype=dtype, device="cuda")
    moved = buf[1:1 + o.numel()].view(o.shape)
    moved.copy_(o)
    assert moved.data_ptr() % 16 != 0
    want = F.conv_headmix_backward(q, k, v, w, o, do, l, m, th, True, 0.125)
    got = F.conv_headmix_backward(q, k, v, w, moved, do, l, m, th, True, 0.125)
    assert all((a is None and b is None) or torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("name", ["conv", "mix", "conv_mix"])
def test_saved_tensors_may_come_back_anywhere(name):
    """Saved-tensor hooks may give the backward copies of what it saved, on other addresses."""
    op = _ops()[name]

    def unpack(t):
        if t.dtype == torch.bfloat16:            # operands of the tensor cores: 16-byte boundaries, as everywhere
            return t.clone()
        buf = torch.zeros(t.numel() + 4, dtype=t.dtype, device="cuda")
        buf[1:1 + t.numel()].view(t.shape).copy_(t)
        return buf[1:1 + t.numel()].view(t.shape)

    grads = []
    for hooks in (False, True):
        args = [t.clone().requires_grad_() for t in _inputs(5)]
        wrt = [t for t, used in zip(args, (1, 1, 1, name != "mix", name != "conv")) if used]
        if hooks:
            with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
                o = op(*args)
        else:
            o = op(*args)
        grads.append(torch.autograd.grad(o, wrt, torch.ones_like(o)))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_exact_kernels_chosen_between_forward_and_backward():
    """The process-wide choice of kernels holds for a backward whose forward ran before it."""
    import fmta_b200 as F
    from fmta_b200._lib import lib
    q, k, v, theta, _ = _inputs(6)
    scale, do = 0.125, torch.randn(q.shape, device="cuda")
    args = [t.clone().requires_grad_() for t in (q, k, v, theta)]
    o = F.FlashConvAttentionCUDAFunction.apply(*args, scale, 2, 2, True)
    old = lib.fmta_set_path(0)
    try:
        got = torch.autograd.grad(o, args, do)
    finally:
        lib.fmta_set_path(old)
    from fmta_b200 import conv_attn
    O, M, L, LSE = conv_attn.forward(q, k, v, theta, scale, 2, 2, True, return_lse=True)
    assert torch.equal(O, o)
    dob = do.to(torch.bfloat16)
    want = conv_attn.backward(q, k, v, dob, conv_attn.rowdot(dob, O), LSE, theta, scale, 2, 2, True, path=0)
    assert all(torch.equal(a, b.to(a.dtype)) for a, b in zip(got, want))


@pytest.mark.parametrize("name", ["mix", "conv", "conv_mix", "conv_kept_keys"])
def test_first_call_of_a_thread(name):
    """A thread whose first use of the GPU is this call (its memory comes from the allocator's cache)."""
    import fmta_b200 as F
    from fmta_b200 import conv_attn
    q, k, v, theta, w = _inputs(8)
    kt = conv_attn.ktilde_buffer(q, theta)
    ops = dict(_ops(), conv_kept_keys=lambda q, k, v, t, w: conv_attn.forward(q, k, v, t, 0.125, 2, 2, True, ktilde=kt)[0])

    def call(out):
        with torch.no_grad():
            out.append(ops[name](q, k, v, theta, w))

    want, got = [], []
    call(want)
    call(want)
    torch.cuda.synchronize()
    worker = threading.Thread(target=call, args=(got,))
    worker.start()
    worker.join()
    assert len(got) == 1 and torch.equal(got[0], want[0])


@pytest.mark.parametrize("name", ["conv", "mix", "decode"])
def test_other_threads_run_while_a_launch_waits(name):
    """A call that waits for room in the GPU's launch queue does not hold the interpreter."""
    import fmta_b200 as F
    q, k, v, theta, w = _inputs(7)
    ops = dict(_ops(), decode=lambda q, k, v, t, w: F.forward_inference(q[:, :, :3].contiguous(), k, v, t, 1, 0.1, 2, 2, False))

    def call():
        with torch.no_grad():
            ops[name](q, k, v, theta, w)

    call()
    torch.cuda.synchronize()
    took = []

    def fill():
        t0 = time.perf_counter()
        for _ in range(2500):
            call()
        took.append(time.perf_counter() - t0)

    torch.cuda._sleep(3_000_000_000)            # about 1.6 s on the GPU: everything behind it queues up
    worker = threading.Thread(target=fill)
    worker.start()
    gap, last = 0.0, time.perf_counter()
    while worker.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    worker.join()
    torch.cuda.synchronize()
    assert took[0] > 1.0                        # the queue did fill
    assert gap < 0.3


@pytest.mark.parametrize("keep,kept", [(False, 0), (None, 1), (True, 1)])
def test_stacked_keys_are_kept_as_asked(monkeypatch, keep, kept):
    from fmta_b200 import conv_attn
    monkeypatch.setattr(conv_attn, "KEEP_KTILDE", keep)
    q, k, v, theta, w = _inputs(9)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.dim()), t)[1], lambda t: t):
        _ops()["conv"](q.requires_grad_(), k, v, theta, w)
    assert seen.count(5) == kept                # [B, H, c_q, N, d]
