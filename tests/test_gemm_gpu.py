"""tcgen05 GEMM family vs. a plain PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    B = b.float().t() if b_mn else b.float()
    return A @ B.t()


def _close(out, ref, k):
    tol = 2e-2 * max(1.0, (k ** 0.5) / 8)
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err <= tol * scale / 4 + 1e-2, f"max err {err} (scale {scale})"
    # the element-wise bound above only catches mis-indexed tiles; a dropped k-slice at large K changes
    # every element a little, which the relative Frobenius error sees (bf16 output rounding alone
    # gives about 1.7e-3)
    fro = ((out.float() - ref).norm() / (ref.norm() + 1e-12)).item()
    assert fro <= 4e-3, f"relative Frobenius error {fro}"


def _route(m, n, k, a_mn, b_mn, split=1, workspace=0):
    """(tile shape, slices of K) that a plain product takes; no operand is looked at."""
    import ctypes
    from neuralfn_b200.ops import _lib
    a, slices = _lib.GemmArgs(), ctypes.c_int()
    a.m, a.n, a.k, a.lda, a.ldb, a.ldc = m, n, k, m if a_mn else k, n if b_mn else k, n
    a.a_mn, a.b_mn, a.alpha, a.split_k, a.workspace, a.workspace_bytes = int(a_mn), int(b_mn), 1.0, split, 256 if workspace else None, workspace
    return ("128", "256", "pair", "cluster")[_lib.load().nfn_gemm_plan(ctypes.byref(a), ctypes.byref(slices))], slices.value


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 256, 128), (384, 768, 768), (1000, 264, 200),
                                   (4096, 2304, 768), (2048, 50304, 768)])
def test_gemm_layouts(kernel_lib, a_mn, b_mn, m, n, k):
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    if a_mn and m % 8:
        pytest.skip("MN-major A needs M % 8 == 0")
    torch.manual_seed(0)
    dev = "cuda"
    a = torch.randn((k, m) if a_mn else (m, k), device=dev, dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device=dev, dtype=torch.bfloat16)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    _lib.assert_status_ok("gemm")
    _close(out, _ref(a, b, a_mn, b_mn), k)


def test_gemm_epilogues(kernel_lib):
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    torch.manual_seed(1)
    m, n, k = 512, 768, 256
    x = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(n, k, device="cuda", dtype=torch.bfloat16) * 0.1
    bias = torch.randn(n, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(m, n, device="cuda", dtype=torch.bfloat16)
    base = x.float() @ w.float().t() + bias.float()

    y = gemm(x, w, bias=bias)
    _close(y, base, k)

    pre = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    y = gemm(x, w, bias=bias, act="gelu_tanh", save_pre=pre)
    _close(pre, base, k)
    _close(y, torch.nn.functional.gelu(base, approximate="tanh"), k)

    y = gemm(x, w, bias=bias, act="gelu_erf")
    _close(y, torch.nn.functional.gelu(base), k)

    y = gemm(x, w, bias=bias, resid=res)
    _close(y, base + res.float(), k)

    # dGELU epilogue: (x @ w.T) * gelu'(pre)
    pre_f = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(pre_f, approximate="tanh").sum().backward()
    y = gemm(x, w, act="gelu_tanh", dact_pre=pre)
    _close(y, (x.float() @ w.float().t()) * pre_f.grad, k)

    # fp32 output with accumulation
    acc = torch.ones(m, n, device="cuda", dtype=torch.float32)
    gemm(x, w, out=acc, accum=True, alpha=0.5)
    _close(acc, 0.5 * (x.float() @ w.float().t()) + 1.0, k)

    # logit soft-cap
    y = gemm(x, w, act="tanh_cap", act_param=30.0)
    _close(y, 30.0 * torch.tanh((x.float() @ w.float().t()) / 30.0), k)
    _lib.assert_status_ok("gemm epilogues")


def test_gemm_strided_views(kernel_lib):
    """Operands that are column slices of a wider buffer (leading dim > width)."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    torch.manual_seed(2)
    big = torch.randn(256, 3 * 128, device="cuda", dtype=torch.bfloat16)
    x = big[:, 128:256]
    w = torch.randn(64, 128, device="cuda", dtype=torch.bfloat16)
    outbuf = torch.zeros(256, 256, device="cuda", dtype=torch.bfloat16)
    out = outbuf[:, 64:128]
    gemm(x, w, out=out)
    _lib.assert_status_ok("gemm views")
    _close(out, x.float() @ w.float().t(), 128)
    assert outbuf[:, :64].abs().max().item() == 0 and outbuf[:, 128:].abs().max().item() == 0


@pytest.mark.parametrize("m,n,k", [(16384, 768, 768), (16384, 2304, 768), (8192, 3072, 768), (16384, 768, 3072),
                                   (8192 + 128, 2304 + 64, 768 + 32)])
def test_gemm_cta_pair(kernel_lib, m, n, k):
    """CTA-pair (cta_group::2) kernel: plain product and the fused epilogues against fp32."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    L = _lib.load()
    torch.manual_seed(3)
    x = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(n, k, device="cuda", dtype=torch.bfloat16) * 0.05
    bias = torch.randn(n, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(m, n, device="cuda", dtype=torch.bfloat16)
    base = x.float() @ w.float().t()
    old = L.nfn_gemm_set_pair_mode(1)
    try:
        y = gemm(x, w)
        _lib.assert_status_ok("gemm pair")
        _close(y, base, k)
        pre = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
        y = gemm(x, w, bias=bias, act="gelu_tanh", save_pre=pre)
        _lib.assert_status_ok("gemm pair gelu")
        _close(pre, base + bias.float(), k)
        _close(y, torch.nn.functional.gelu(base + bias.float(), approximate="tanh"), k)
        y = gemm(x, w, bias=bias, resid=res)
        _lib.assert_status_ok("gemm pair resid")
        _close(y, base + bias.float() + res.float(), k)
    finally:
        L.nfn_gemm_set_pair_mode(old)


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(4096, 4096), (1000, 1032), (6144, 14336)])
def test_gemv_small_m_with_epilogues(kernel_lib, m, n, k):
    """Products with at most four rows take the weight-streaming GEMV kernel; same epilogue semantics
    as the tensor-core path (checked against fp32 and against the GEMM path itself)."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    torch.manual_seed(m * 7 + n)
    a = (torch.randn(m, k, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    bias = (torch.randn(n, device="cuda") * 0.1).bfloat16()
    resid = torch.randn(m, n, device="cuda").bfloat16()
    ref = a.float() @ w.float().t()
    _close(gemm(a, w), ref, k)
    out = gemm(a, w, bias=bias, act="gelu_tanh", resid=resid)
    full = torch.nn.functional.gelu(ref + bias.float(), approximate="tanh") + resid.float()
    _close(out, full, k)
    acc = resid.clone()
    gemm(a, w, out=acc, accum=True, alpha=0.5)
    _close(acc, resid.float() + 0.5 * ref, k)
    capped = gemm(a, w, act="tanh_cap", act_param=2.0)
    _close(capped, 2.0 * torch.tanh(ref / 2.0), k)
    # the tensor-core path gives the same numbers
    L = _lib.load()
    old = L.nfn_gemm_set_gemv_mode(0)
    try:
        tc = gemm(a, w, bias=bias, act="gelu_tanh", resid=resid)
    finally:
        L.nfn_gemm_set_gemv_mode(old)
    torch.testing.assert_close(out.float(), tc.float(), atol=3e-2, rtol=3e-2)
    _lib.assert_status_ok("gemv")


@pytest.mark.parametrize("m,n,k", [(16384, 768, 2304), (16384, 3072, 768), (8192 + 128, 768 + 64, 3072 + 32), (1024, 256, 256)])
def test_gemm_cta_pair_mn_major_b(kernel_lib, m, n, k):
    """CTA-pair kernel with an MN-major B operand (input gradients dY W): plain product and the
    dGELU epilogue against fp32; the one-CTA kernel must agree to rounding."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    L = _lib.load()
    torch.manual_seed(5)
    dy = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(k, n, device="cuda", dtype=torch.bfloat16) * 0.05      # [K, N]: N contiguous
    pre = torch.randn(m, n, device="cuda", dtype=torch.bfloat16)
    base = dy.float() @ w.float()
    t = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(t, approximate="tanh").sum().backward()
    old = L.nfn_gemm_set_pair_mode(1)
    try:
        y = gemm(dy, w, b_mn=True)
        _lib.assert_status_ok("gemm pair b_mn")
        _close(y, base, k)
        yg = gemm(dy, w, b_mn=True, act="gelu_tanh", dact_pre=pre)
        _lib.assert_status_ok("gemm pair b_mn dgelu")
        _close(yg, base * t.grad, k)
        L.nfn_gemm_set_pair_mode(0)
        y1 = gemm(dy, w, b_mn=True)
        assert (y.float() - y1.float()).abs().max().item() <= 0.02 * base.abs().max().item()
    finally:
        L.nfn_gemm_set_pair_mode(old)


@pytest.mark.parametrize("m", [3, 8, 17, 32, 33, 64])
@pytest.mark.parametrize("n,k", [(6656, 1024), (2304, 6656), (1000, 1056)])
def test_skinny_products_take_the_weight_streaming_mma_kernel(kernel_lib, m, n, k):
    """3 - 64 rows over a large K-major weight matrix: mma.sync with permuted-k fragments, in-CTA split-K, fused epilogue.
    Checked against fp32 and against the tcgen05 split-K path it replaces."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    torch.manual_seed(m * 13 + n)
    a = (torch.randn(m, k, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    bias = (torch.randn(n, device="cuda") * 0.1).bfloat16()
    resid = torch.randn(m, n, device="cuda").bfloat16()
    ws = torch.empty(32 * 1024 * 1024, device="cuda", dtype=torch.float32)
    L = _lib.load()
    forced = L.nfn_gemm_skinny_set_impl(2)                         # every eligible row count (the default stops at 16 rows)
    before = _lib.launch_count()
    ref = a.float() @ w.float().t()
    y = gemm(a, w, workspace=ws)
    assert _lib.launch_count() - before == 1                       # one launch: no separate split-K reduction
    _close(y, ref, k)
    out = gemm(a, w, bias=bias, act="silu", resid=resid, workspace=ws)
    _close(out, torch.nn.functional.silu(ref + bias.float()) + resid.float(), k)
    acc = resid.clone()
    gemm(a, w, out=acc, accum=True, alpha=0.5, workspace=ws)
    _close(acc, resid.float() + 0.5 * ref, k)
    # strided views: rows of a wider buffer in, columns of a wider buffer out
    wide_in = torch.zeros(m, k + 64, device="cuda", dtype=torch.bfloat16)
    wide_in[:, :k] = a
    wide_out = torch.zeros(m, n + 128, device="cuda", dtype=torch.bfloat16)
    gemm(wide_in[:, :k], w, out=wide_out[:, 64:64 + n], workspace=ws)
    _close(wide_out[:, 64:64 + n], ref, k)
    assert float(wide_out[:, :64].abs().max()) == 0.0 and float(wide_out[:, 64 + n:].abs().max()) == 0.0
    L.nfn_gemm_skinny_set_impl(0)
    try:
        tc = gemm(a, w, bias=bias, act="silu", resid=resid, workspace=ws)
    finally:
        L.nfn_gemm_skinny_set_impl(forced)
    torch.testing.assert_close(out.float(), tc.float(), atol=4e-2, rtol=4e-2)
    _lib.assert_status_ok("skinny gemm")


@pytest.mark.parametrize("m,mode", [(17, 3), (24, 3), (32, 3), (5, 3), (16, 3)])
@pytest.mark.parametrize("n,k", [(6656, 1024), (2304, 6656), (1000, 1056), (12288, 6656), (520, 4096)])
def test_skinny_products_with_resident_token_fragments(kernel_lib, m, mode, n, k):
    """The opt-in form for up to 32 rows: token fragments held in registers, K split over a thread-block cluster whose CTAs
    add their strips over distributed shared memory. One launch, the same bits on every call, fp32 and tcgen05 agreement."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    torch.manual_seed(m * 7 + n)
    a = (torch.randn(m, k, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    bias = (torch.randn(n, device="cuda") * 0.1).bfloat16()
    resid = torch.randn(m, n, device="cuda").bfloat16()
    ws = torch.empty(32 * 1024 * 1024, device="cuda", dtype=torch.float32)
    L = _lib.load()
    old = L.nfn_gemm_skinny_set_impl(mode)
    try:
        ref = a.float() @ w.float().t()
        before = _lib.launch_count()
        y = gemm(a, w, workspace=ws)
        assert _lib.launch_count() - before == 1
        _close(y, ref, k)
        assert torch.equal(y, gemm(a, w, workspace=ws))
        out = gemm(a, w, bias=bias, act="gelu_tanh", resid=resid, workspace=ws)
        _close(out, torch.nn.functional.gelu(ref + bias.float(), approximate="tanh") + resid.float(), k)
        acc = resid.clone()
        gemm(a, w, out=acc, accum=True, alpha=0.5, workspace=ws)
        _close(acc, resid.float() + 0.5 * ref, k)
        wide_in = torch.zeros(m, k + 64, device="cuda", dtype=torch.bfloat16)
        wide_in[:, :k] = a
        wide_out = torch.zeros(m, n + 128, device="cuda", dtype=torch.bfloat16)
        gemm(wide_in[:, :k], w, out=wide_out[:, 64:64 + n], workspace=ws)
        _close(wide_out[:, 64:64 + n], ref, k)
        assert float(wide_out[:, :64].abs().max()) == 0.0 and float(wide_out[:, 64 + n:].abs().max()) == 0.0
        L.nfn_gemm_skinny_set_impl(0)
        tc = gemm(a, w, bias=bias, act="gelu_tanh", resid=resid, workspace=ws)
    finally:
        L.nfn_gemm_skinny_set_impl(old)
    torch.testing.assert_close(out.float(), tc.float(), atol=4e-2, rtol=4e-2)
    _lib.assert_status_ok("resident skinny gemm")


@pytest.mark.parametrize("m,n,dtype", [(256, 512, torch.bfloat16), (2048, 1024, torch.bfloat16), (192, 200, torch.float32)])
def test_grouped_contraction_gives_every_experts_weight_gradient(kernel_lib, m, n, dtype):
    """out[g] = a[rows of g]^T b[rows of g] for all groups in one launch: segments padded to 128 rows with zero rows in a, an empty
    group, accumulation on top of an existing gradient."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm_grouped_k
    torch.manual_seed(m + n)
    counts = [300, 0, 128, 77, 1, 513]
    offs = [0]
    for c in counts:
        offs.append(offs[-1] + (c + 127) // 128 * 128)
    rows = offs[-1] + 256                                             # rows past the last group are never read
    a = torch.zeros(rows, m, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(rows, n, device="cuda") * 0.3).bfloat16()        # padding rows of b are finite, not zero
    for g, c in enumerate(counts):
        a[offs[g]:offs[g] + c] = (torch.randn(c, m, device="cuda") * 0.3).bfloat16()
    a[offs[-1]:] = float("nan")                                       # must not be touched
    group_rows = torch.tensor(offs, device="cuda", dtype=torch.int32)
    out = torch.full((len(counts), m, n), 7.0, device="cuda", dtype=dtype)
    before = _lib.launch_count()
    gemm_grouped_k(a, b, group_rows, out)
    assert _lib.launch_count() - before == 1
    ref = torch.stack([a[offs[g]:offs[g] + c].float().t() @ b[offs[g]:offs[g] + c].float() for g, c in enumerate(counts)])
    assert float(out[1].abs().max()) == 0.0
    tol = 2e-2 * float(ref.abs().max()) + 1e-3
    assert float((out.float() - ref).abs().max()) < tol
    keep = out.clone()
    gemm_grouped_k(a, b, group_rows, out, alpha=0.5, accum=True)
    assert float((out.float() - (keep.float() + 0.5 * ref)).abs().max()) < 2 * tol
    # column views of a wider buffer (the gate / up halves of the hidden gradient)
    wide = torch.zeros(rows, 2 * n, device="cuda", dtype=torch.bfloat16)
    wide[:, n:] = b
    out2 = torch.empty_like(keep)
    gemm_grouped_k(a, wide[:, n:], group_rows, out2)
    assert torch.equal(out2, keep)
    _lib.assert_status_ok("grouped contraction")


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("m,n,k,split,route", [
    (2056, 2312, 72, 1, ("128", 1)), (6664, 776, 1000, 1, ("pair", 1)), (264, 520, 4104, 5, ("128", 5)), (776, 264, 16392, 0, ("cluster", 6)),
    (136, 19208, 520, 1, ("pair", 1)), (1032, 1288, 8200, 0, ("pair", 2)), (2056, 2312, 4104, 2, ("pair", 2)), (776, 1288, 16392, 0, ("pair", 3)),
    (520, 2056, 8200, 0, ("256", 3)), (4104, 1032, 1000, 5, ("pair", 1))])
def test_gemm_pairs_and_slices_at_edges(kernel_lib, a_mn, b_mn, m, n, k, split, route):
    """Remainders of every tile shape and of the k-block, an uneven last slice, slices on CTA pairs, slices that the
    workspace does not hold, in all four operand layouts; equal results on every run."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    assert _route(m, n, k, a_mn, b_mn, split=split, workspace=64 << 20) == route
    torch.manual_seed(m)
    a = torch.randn((k, m) if a_mn else (m, k), device="cuda", dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda", dtype=torch.bfloat16)
    ws = torch.empty(64 << 20, device="cuda", dtype=torch.uint8)
    guard = torch.full((m + 1, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=guard[:m, :n], workspace=ws, split_k=split)
    again = gemm(a, b, a_mn=a_mn, b_mn=b_mn, workspace=ws, split_k=split)
    _lib.assert_status_ok("gemm")
    _close(out, _ref(a, b, a_mn, b_mn), k)
    assert torch.equal(out, again) and bool((guard[m:] == 7).all()) and bool((guard[:, n:] == 7).all())


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("m,n,k", [(136, 128, 520), (256, 264, 1032), (24, 2056, 4104), (520, 136, 6000), (136, 128, 2056), (130, 136, 4104)])
def test_gemm_slices_in_a_cluster(kernel_lib, a_mn, b_mn, m, n, k):
    """Fewer tiles than SMs: K cut over a cluster (uneven slices, remainders of tile and k-block, two rows of a tile for more ranks), with every epilogue;
    the first shape has too short a K and takes whole tiles."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    if a_mn and m % 8:
        pytest.skip("MN-major A needs M % 8 == 0")
    tile, slices = _route(m, n, k, a_mn, b_mn)
    assert tile == ("128" if k < 1000 else "cluster") and (m != 130 or slices > m % 128)
    torch.manual_seed(m)
    dev = "cuda"
    a = torch.randn((k, m) if a_mn else (m, k), device=dev, dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device=dev, dtype=torch.bfloat16)
    bias, res = torch.randn(n, device=dev).bfloat16(), torch.randn(m, n, device=dev).bfloat16()
    base = _ref(a, b, a_mn, b_mn)
    guard = torch.full((m + 1, n + 8), 7.0, device=dev, dtype=torch.bfloat16)
    _close(gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=guard[:m, :n]), base, k)
    assert bool((guard[m:] == 7).all()) and bool((guard[:, n:] == 7).all())
    _close(gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, resid=res), base + bias.float() + res.float(), k)
    s, pre = 1.0 / k ** 0.5, torch.empty(m, n, device=dev, dtype=torch.bfloat16)
    y = gemm(a, b, a_mn=a_mn, b_mn=b_mn, alpha=s, act="gelu_tanh", save_pre=pre, bias=bias)
    _close(pre, base * s + bias.float(), k)
    _close(y, torch.nn.functional.gelu(base * s + bias.float(), approximate="tanh"), k)
    z = res.float().requires_grad_(True)
    torch.nn.functional.gelu(z, approximate="tanh").sum().backward()
    _close(gemm(a, b, a_mn=a_mn, b_mn=b_mn, act="gelu_tanh", dact_pre=res), base * z.grad, k)
    c = res.clone()
    _close(gemm(a, b, a_mn=a_mn, b_mn=b_mn, accum=True, out=c), base + res.float(), k)
    f = torch.ones(m, n, device=dev)
    gemm(a, b, a_mn=a_mn, b_mn=b_mn, accum=True, out=f)
    _close(f, base + 1, k)
    _lib.assert_status_ok("gemm slices")


@pytest.mark.parametrize("m,ff,k", [(8191, 1048, 512), (4100, 3000, 1032), (2056, 11272, 520), (1, 136, 64), (2, 1000, 5640), (1, 5632, 2048), (2, 136, 8200)])
def test_gemm_swiglu(kernel_lib, m, ff, k):
    """Gate and up of a column in one pair tile: a last column tile that runs from the gates into the ups, row and k remainders;
    gate and up row of a warp pair for one and two rows, at each number of warps that share it. One rounding to bf16 of
    fp32 values."""
    import ctypes
    from neuralfn_b200.ops import _lib
    torch.manual_seed(m)
    x, w = torch.randn(m, k, device="cuda").bfloat16(), (torch.randn(2 * ff, k, device="cuda") * k ** -0.5).bfloat16()
    out = torch.full((m + 1, ff + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    P, I = ctypes.c_void_p, ctypes.c_int
    rc = _lib.load().nfn_gemm_swiglu(P(x.data_ptr()), I(k), P(w.data_ptr()), I(k), P(out.data_ptr()), I(ff + 8), I(m), I(ff), I(k), I(0), P(_lib.stream_ptr()))
    assert rc == 1
    g, u = (x.double() @ w.double().T).split(ff, -1)
    ref = torch.nn.functional.silu(g) * u
    _lib.assert_status_ok("gemm_swiglu")
    assert bool(((out[:m, :ff].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all())
    assert bool((out[m:] == 7).all()) and bool((out[:, ff:] == 7).all())


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("m,n,k", [(96, 264, 1032), (264, 520, 4104), (2056, 2312, 1032)])
@pytest.mark.parametrize("split", [2, 5])
def test_gemm_with_given_slices_keeps_its_epilogue(kernel_lib, a_mn, b_mn, m, n, k, split):
    """A number of K slices given together with an epilogue that slices cannot carry: the product runs with that epilogue. Plain, accumulating and
    scaled products take the slices."""
    from neuralfn_b200.ops import _lib
    from neuralfn_b200.ops.gemm import gemm
    torch.manual_seed(m + split)
    dev = "cuda"
    a = torch.randn((k, m) if a_mn else (m, k), device=dev, dtype=torch.bfloat16)
    b = torch.randn((k, n) if b_mn else (n, k), device=dev, dtype=torch.bfloat16)
    bias, res = torch.randn(n, device=dev).bfloat16(), torch.randn(m, n, device=dev).bfloat16()
    s = k ** -0.5
    base = _ref(a, b, a_mn, b_mn) * s
    gelu = lambda t: torch.nn.functional.gelu(t, approximate="tanh")  # noqa: E731
    ws = torch.empty(5 * m * n * 4, device=dev, dtype=torch.uint8)
    run = lambda **kw: gemm(a, b, a_mn=a_mn, b_mn=b_mn, alpha=s, workspace=ws, split_k=split, **kw)  # noqa: E731
    _close(run(), base, 64)
    _close(run(accum=True, out=res.clone()), base + res.float(), 64)
    _close(run(bias=bias), base + bias.float(), 64)
    _close(run(resid=res), base + res.float(), 64)
    _close(run(act="gelu_tanh"), gelu(base), 64)
    pre = torch.zeros(m, n, device=dev, dtype=torch.bfloat16)
    _close(run(bias=bias, act="gelu_tanh", save_pre=pre), gelu(base + bias.float()), 64)
    _close(pre, base + bias.float(), 64)
    z = res.float().requires_grad_(True)
    gelu(z).sum().backward()
    _close(run(act="gelu_tanh", dact_pre=res), base * z.grad, 64)
    _lib.assert_status_ok("gemm slices with an epilogue")
