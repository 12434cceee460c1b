"""Mixture-of-experts forward (routing, permutation, grouped GEMMs, combine) vs the fp32 oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k,d,F,score", [(300, 8, 2, 256, 512, "softmax"), (1000, 64, 8, 512, 256, "sigmoid"), (17, 4, 1, 128, 128, "softmax")])
def test_moe_forward_matches_reference(T, E, k, d, F, score):
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.moe import MoEWorkspace, moe_forward, moe_reference
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    x = (torch.randn(T, d, device=dev) * 0.5).bfloat16()
    wr = (torch.randn(E, d, device=dev) * 0.2).bfloat16()
    wgu = (torch.randn(E, 2 * F, d, device=dev) * 0.05).bfloat16()
    wd = (torch.randn(E, d, F, device=dev) * 0.05).bfloat16()
    resid = torch.randn(T, d, device=dev).bfloat16()
    ws = MoEWorkspace(T, E, k, d, F, dev)
    for _ in range(2):  # second call reuses the workspace (counters must be clean again)
        out = moe_forward(x, wr, wgu, wd, k, ws, score_fn=score, resid=resid)
    torch.cuda.synchronize()
    assert _lib.status_read_reset() == 0
    ref = moe_reference(x, wr, wgu, wd, k, score_fn=score, resid=resid)
    # routing decisions are made on fp32 logits of bf16 inputs on both sides; a near-tie may
    # still flip an expert for a token, so compare per-token and allow a handful of outliers
    err = (out.float() - ref).abs().amax(-1)
    assert float((err > 0.08).float().mean()) < 0.02, float(err.max())
    assert int(ws.plan[0]) * 128 == int(ws.plan[1]) and int(ws.counts.sum()) == T * k


@pytest.mark.gpu
@pytest.mark.parametrize("E,k,T", [(8, 2, 300), (16, 4, 1024)])
def test_moe_experts_autograd_matches_torch(E, k, T):
    """Native expert FFN with gradients against the per-expert PyTorch loop in fp32."""
    import neuralfn_b200.tensor.stages_moe as SM
    from neuralfn_b200.ops.moe import moe_experts
    d, h = 256, 384
    g = torch.Generator(device="cuda").manual_seed(E * 100 + k)
    x = torch.randn(T, d, device="cuda", generator=g)
    w1, w3 = (torch.randn(E, d, h, device="cuda", generator=g) * 0.05 for _ in range(2))
    w2 = torch.randn(E, h, d, device="cuda", generator=g) * 0.05
    logits = torch.randn(T, E, device="cuda", generator=g)
    wts, idx = torch.softmax(logits, -1).topk(k, -1)
    wts = wts / wts.sum(-1, keepdim=True)
    dout = torch.randn(T, d, device="cuda", generator=g)

    ref_in = [t.clone().requires_grad_(True) for t in (x, w1, w2, w3, wts)]
    SM._FORCE_TORCH_MOE = True
    try:
        ref = SM.grouped_swiglu_experts(ref_in[0], ref_in[1], ref_in[2], ref_in[3], ref_in[4], idx)
    finally:
        SM._FORCE_TORCH_MOE = False
    ref.backward(dout)

    got_in = [t.to(torch.bfloat16).requires_grad_(True) for t in (x, w1, w2, w3)] + [wts.clone().requires_grad_(True)]
    got = moe_experts(got_in[0], got_in[1], got_in[2], got_in[3], got_in[4], idx)
    got.backward(dout.to(torch.bfloat16))

    def rel(a, b):
        return float((a.float() - b.float()).abs().max() / (b.float().abs().max() + 1e-9))

    assert rel(got, ref) < 0.03
    for name, a, b in zip(("dx", "dw1", "dw2", "dw3", "dweights"), got_in, ref_in):
        assert rel(a.grad, b.grad) < 0.04, (name, rel(a.grad, b.grad))

    # the stage function takes the native path for bf16 CUDA tensors
    y = SM.grouped_swiglu_experts(got_in[0].detach(), got_in[1].detach(), got_in[2].detach(), got_in[3].detach(), wts, idx)
    assert y.dtype == torch.bfloat16 and rel(y, ref) < 0.03


@pytest.mark.gpu
@pytest.mark.parametrize("T,d,h,E,k,used", [
    (1, 64, 64, 1, 1, 1),            # one row, one expert
    (17, 64, 192, 4, 1, 2),          # a column tile that straddles the end of the hidden width, experts without rows
    (129, 192, 320, 8, 8, 8),        # every expert for every token, widths that fill no tile
    (1000, 512, 256, 256, 2, 256),   # the most experts
    (2500, 256, 1088, 3, 3, 3),      # wide tiles, a remainder of the last one
])
def test_moe_experts_against_64_bit(kernel_lib, T, d, h, E, k, used):
    """Results and gradients are within a few roundings to bf16 (2^-9 each) of the 64-bit values of the same bf16 inputs: rows pass three of
    them (gate and up, their product, the output), gradients four; 2-norms average them, so 3e-3 per rounding is a bound."""
    from neuralfn_b200.ops.moe import moe_experts
    g = torch.Generator(device="cuda").manual_seed(T + h)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x, w1, w2, w3, dout = r(T, d).bfloat16(), (r(E, d, h) * 0.05).bfloat16(), (r(E, h, d) * 0.05).bfloat16(), (r(E, d, h) * 0.05).bfloat16(), r(T, d).bfloat16()
    wt, idx = torch.softmax(r(T, used), -1).topk(k, -1)
    got_in = [t.clone().requires_grad_(True) for t in (x, w1, w2, w3, wt)]
    got = moe_experts(*got_in, idx)
    grads = torch.autograd.grad(got, got_in, dout)
    ref_in = [t.double().requires_grad_(True) for t in (x, w1, w2, w3, wt)]
    out = torch.zeros(T, d, dtype=torch.float64, device="cuda")
    for e in range(used):
        rows, place = (idx == e).nonzero(as_tuple=True)
        y = (torch.nn.functional.silu(ref_in[0][rows] @ ref_in[1][e]) * (ref_in[0][rows] @ ref_in[3][e])) @ ref_in[2][e]
        out = out.index_add(0, rows, y * ref_in[4][rows, place][:, None])
    want = torch.autograd.grad(out, ref_in, dout.double())
    for name, a, b in zip(("out", "dx", "dw1", "dw2", "dw3", "dweights"), (got, *grads), (out, *want)):
        assert float((a.double() - b).norm()) <= 0.012 * float(b.norm()) + 1e-12, name
    again = moe_experts(*got_in, idx)
    assert torch.equal(again, got) and all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(again, got_in, dout), grads))


@pytest.mark.gpu
def test_moe_experts_refuses_an_expert_that_is_not_there(kernel_lib):
    from neuralfn_b200.ops.moe import moe_experts
    w = torch.zeros(4, 64, 64, device="cuda", dtype=torch.bfloat16)
    x, wt = torch.zeros(3, 64, device="cuda", dtype=torch.bfloat16), torch.ones(3, 1, device="cuda")
    for bad in (-1, 4):
        with pytest.raises(RuntimeError):
            moe_experts(x, w, w, w, wt, torch.tensor([[0], [bad], [1]], device="cuda"))
    moe_experts(x, w, w, w, wt, torch.tensor([[0], [3], [1]], device="cuda"))


def _experts_case(T, d, h, E, k, seed, index_dtype=torch.int64):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    t = [r(T, d).bfloat16(), (r(E, d, h) * 0.05).bfloat16(), (r(E, h, d) * 0.05).bfloat16(), (r(E, d, h) * 0.05).bfloat16()]
    wt, idx = torch.softmax(r(T, E), -1).topk(k, -1)
    return t, wt, idx.to(index_dtype), r(T, d).bfloat16()


def test_moe_experts_takes_weights_and_indices_as_they_come(kernel_lib):
    """One weight per token, indices of another whole-number type, either of them on the host: the values of the full device tensors."""
    from neuralfn_b200.ops.moe import moe_experts
    t, wt, idx, dout = _experts_case(130, 64, 192, 8, 3, 5)
    one = wt[:, :1].clone().requires_grad_(True)
    want_in = wt[:, :1].expand(-1, 3).clone().requires_grad_(True)
    want = moe_experts(*t, want_in, idx)
    got = moe_experts(*t, one, idx)
    assert torch.equal(got, want)
    torch.testing.assert_close(torch.autograd.grad(got, one, dout)[0], torch.autograd.grad(want, want_in, dout)[0].sum(1, keepdim=True))
    full = moe_experts(*t, wt, idx)
    for w, i in ((wt, idx.int()), (wt, idx.cpu()), (wt.cpu(), idx), (wt.double(), idx.short())):
        assert torch.equal(moe_experts(*t, w, i), full)


def _experts_exact(t, wt, idx):
    x, w1, w2, w3 = (v.double() for v in t)
    out = torch.zeros_like(x)
    for e in range(w1.shape[0]):
        rows, place = (idx == e).nonzero(as_tuple=True)
        y = (torch.nn.functional.silu(x[rows] @ w1[e]) * (x[rows] @ w3[e])) @ w2[e]
        out = out.index_add(0, rows, y * wt.double()[rows, place][:, None])
    return out


@pytest.mark.parametrize("T,d,h,E,k", [(50, 72, 40, 4, 2), (33, 64, 72, 3, 1), (40, 136, 64, 6, 3), (129, 64, 64, 16, 9), (7, 64, 128, 32, 32)])
def test_moe_experts_of_other_widths_and_counts(kernel_lib, T, d, h, E, k):
    """Widths that are multiples of eight only, more than eight experts per token: within the roundings to bf16 (see above) of the 64-bit values."""
    from neuralfn_b200.ops.moe import moe_experts
    t, wt, idx, dout = _experts_case(T, d, h, E, k, T + d)
    got_in = [v.clone().requires_grad_(True) for v in (*t, wt)]
    got = moe_experts(*got_in, idx)
    grads = torch.autograd.grad(got, got_in, dout)
    ref_in = [v.double().requires_grad_(True) for v in (*t, wt)]
    out = _experts_exact(ref_in[:4], ref_in[4], idx)
    want = torch.autograd.grad(out, ref_in, dout.double())
    for name, a, b in zip(("out", "dx", "dw1", "dw2", "dw3", "dweights"), (got, *grads), (out, *want)):
        assert float((a.double() - b).norm()) <= 0.012 * float(b.norm()) + 1e-12, name


def test_moe_experts_without_tokens(kernel_lib):
    from neuralfn_b200.ops.moe import moe_experts
    t, wt, idx, dout = _experts_case(0, 64, 128, 4, 2, 0)
    got_in = [v.clone().requires_grad_(True) for v in (*t, wt)]
    got = moe_experts(*got_in, idx)
    grads = torch.autograd.grad(got, got_in, dout)
    assert got.shape == (0, 64) and all(a.shape == b.shape and not bool(a.any()) for a, b in zip(grads, got_in))


def test_moe_experts_in_a_graph(kernel_lib):
    """Captured forward and backward on a thread whose first expert call this is, replayed on other inputs: the values of the eager call. An expert that is
    not there leaves its entry out of the replay."""
    import threading
    from neuralfn_b200.ops.moe import moe_experts
    t, wt, idx, dout = _experts_case(300, 64, 128, 8, 2, 1)
    t2, wt2, idx2, _ = _experts_case(300, 64, 128, 8, 2, 2)
    leaves = [v.requires_grad_(True) for v in (*t, wt)]
    moe_experts(*leaves, idx)                                       # kernels loaded, attributes set
    torch.cuda.synchronize()
    got, failed = [], []

    def capture():
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                out = moe_experts(*leaves, idx)
                grads = torch.autograd.grad(out, leaves, dout)
            got.extend([graph, out, *grads])
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    worker = threading.Thread(target=capture)
    worker.start()
    worker.join()
    assert not failed, failed
    graph, *results = got
    with torch.no_grad():
        for a, b in zip((*leaves, idx), (*t2, wt2, idx2)):
            a.copy_(b)
    graph.replay()
    torch.cuda.synchronize()
    eager = moe_experts(*leaves, idx)
    for a, b in zip(results, (eager, *torch.autograd.grad(eager, leaves, dout))):
        assert torch.equal(a, b)
    with torch.no_grad():
        idx[5, 1] = 99
    graph.replay()
    torch.cuda.synchronize()
    alone = _experts_exact([v[5:6] if i == 0 else v for i, v in enumerate(leaves[:4])], leaves[4][5:6, :1], idx[5:6, :1])
    assert float((results[0][5].double() - alone[0]).norm()) <= 0.012 * float(alone.norm())
