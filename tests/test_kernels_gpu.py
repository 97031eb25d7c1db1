"""Numerics of every CUDA kernel against a plain PyTorch fp32 statement of the same op (needs a B200)."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf16(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).bfloat16()


def _rel(a, b):
    return ((a.float() - b.float()).abs().max() / b.float().abs().max().clamp(min=1e-6)).item()


@pytest.fixture(autouse=True)
def _seed_and_check():
    torch.manual_seed(0)
    yield
    from pippy_b200.ops import _lib

    _lib.check_device_errors()


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 1)])
def test_gemm_layouts(variant, a_mn, b_mn):
    from pippy_b200.ops.gemm import gemm

    M, N, K = 1000, 776, 520
    a = _bf16(K, M) if a_mn else _bf16(M, K)
    b = _bf16(K, N) if b_mn else _bf16(N, K)
    ref = (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
    out = gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn), variant=variant)
    assert _rel(out, ref) < 1e-2


@pytest.mark.parametrize("variant", [1, 2])
def test_gemm_epilogues(variant):
    from pippy_b200.ops.gemm import gemm

    M, N, K = 512, 768, 256
    a, b = _bf16(M, K), _bf16(N, K)
    bias, res = _bf16(N), _bf16(M, N)
    r0 = a.float() @ b.float().t()
    assert _rel(gemm(a, b, bias=bias, residual=res, variant=variant), r0 + bias.float() + res.float()) < 1e-2
    aux = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, bias=bias, act=1, aux=aux, variant=variant)
    assert _rel(out, F.gelu(r0 + bias.float(), approximate="tanh")) < 1e-2
    assert _rel(aux, r0 + bias.float()) < 1e-2
    acc = torch.ones(M, N, device="cuda")
    gemm(a, b, out=acc, accumulate=True, variant=variant)
    assert _rel(acc, r0 + 1) < 1e-4


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("M,N", [(77, 1000), (300, 256), (257, 288), (33, 40)])
def test_gemm_epilogue_edges(variant, M, N):
    """Rows that end inside a warp's 32, columns that end inside a 32-column chunk, one chunk and odd chunk counts: the
    operands the epilogue fetches ahead (residual, fp32 target) have to belong to the rows and columns it writes."""
    from pippy_b200.ops.gemm import gemm

    K = 192
    a, b, bias, res = _bf16(M, K), _bf16(N, K), _bf16(N), _bf16(M, N)
    r0 = a.float() @ b.float().t()
    assert _rel(gemm(a, b, bias=bias, residual=res, variant=variant), r0 + bias.float() + res.float()) < 1e-2
    acc0 = torch.randn(M + 1, N, device="cuda")  # one guard row
    acc = acc0.clone()
    gemm(a, b, out=acc[:M], accumulate=True, variant=variant)
    assert _rel(acc[:M], acc0[:M] + r0) < 1e-4 and torch.equal(acc[M], acc0[M])
    gemm(a, b, bias=bias, residual=res, out=acc[:M], accumulate=True, variant=variant)
    assert _rel(acc[:M], acc0[:M] + 2 * r0 + bias.float() + res.float()) < 1e-4
    aux = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, bias=bias, residual=res, act=1, aux=aux, variant=variant)
    assert _rel(out, F.gelu(r0 + bias.float(), approximate="tanh") + res.float()) < 1e-2
    assert _rel(aux, r0 + bias.float()) < 1e-2
    aux.fill_(7.0)
    out = gemm(a, b, bias=bias, act=1, aux=aux, variant=variant)
    assert _rel(out, F.gelu(r0 + bias.float(), approximate="tanh")) < 1e-2
    assert _rel(aux, r0 + bias.float()) < 1e-2


@pytest.mark.parametrize("M,N,K", [(77, 4096, 4096), (1, 256, 8192), (700, 1000, 4096), (2048, 768, 16384), (2500, 2600, 8200)])
def test_gemm_split_contraction(M, N, K):
    """Shapes whose last wave is split over ranges of the contraction: the same bits each time, another stream at the same
    time, and a captured call that is replayed beside eager ones."""
    import ctypes

    from pippy_b200.ops import _lib
    from pippy_b200.ops.gemm import gemm

    plan = (ctypes.c_int * 4)()
    _lib.lib().pb_gemm_plan(M, N, K, 148, 1, plan)
    assert plan[2] > 1, list(plan)
    a, b, bias, res = _bf16(M, K), _bf16(K, N), _bf16(N), _bf16(M, N)
    ref = a.float() @ b.float()
    out = gemm(a, b, b_mn=True)
    assert _rel(out, ref) < 1e-2
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        others = [gemm(a, b, b_mn=True) for _ in range(4)]
    again = [gemm(a, b, b_mn=True) for _ in range(4)]
    torch.cuda.current_stream().wait_stream(side)
    assert all(torch.equal(out, o) for o in others + again)
    assert _rel(gemm(a, b, b_mn=True, bias=bias, residual=res), ref + bias.float() + res.float()) < 1e-2
    acc = torch.ones(M, N, device="cuda")
    gemm(a, b, b_mn=True, out=acc, accumulate=True)
    assert _rel(acc, ref + 1) < 1e-4
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = gemm(a, b, b_mn=True)
    for _ in range(2):
        graph.replay()
        assert torch.equal(gemm(a, b, b_mn=True), out)
        assert torch.equal(captured, out)


@pytest.mark.parametrize("M,N,K", [(77, 4096, 4096), (1, 256, 8192), (700, 1000, 4096), (2048, 768, 16384), (2504, 2600, 8200)])
def test_gemm_split_epilogues(M, N, K):
    """Every kind of output of a split tile, an output that is part of a wider buffer, both operands with the contraction
    outside (as in a weight gradient), and a grid with SMs left out."""
    import ctypes

    from pippy_b200.ops import _lib
    from pippy_b200.ops.gemm import gemm, set_sm_reserve

    plan = (ctypes.c_int * 4)()
    _lib.lib().pb_gemm_plan(M, N, K, 148, 1, plan)
    assert plan[2] > 1, list(plan)
    a, b, bias, res = _bf16(M, K), _bf16(K, N), _bf16(N), _bf16(M, N)
    r0 = a.float() @ b.float()
    act = F.gelu(r0 + bias.float(), approximate="tanh")
    aux = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert _rel(gemm(a, b, b_mn=True, bias=bias, act=1, aux=aux), act) < 1e-2 and _rel(aux, r0 + bias.float()) < 1e-2
    aux.zero_()
    assert _rel(gemm(a, b, b_mn=True, bias=bias, residual=res, act=1, aux=aux), act + res.float()) < 1e-2
    assert _rel(aux, r0 + bias.float()) < 1e-2
    assert _rel(gemm(a, b, b_mn=True, act=1), F.gelu(r0, approximate="tanh")) < 1e-2
    assert _rel(gemm(a, b, b_mn=True, out_fp32=True), r0) < 1e-4
    wide = torch.full((M + 1, N + 16), 3.0, device="cuda")
    gemm(a, b, b_mn=True, bias=bias, out=wide[:M, 8 : 8 + N], accumulate=True)
    assert _rel(wide[:M, 8 : 8 + N], r0 + bias.float() + 3) < 1e-4
    assert (wide[M] == 3).all() and (wide[:, :8] == 3).all() and (wide[:, 8 + N :] == 3).all()
    if M % 8 == 0:
        acc = torch.ones(M, N, device="cuda")
        gemm(a.t().contiguous(), b, a_mn=True, b_mn=True, out=acc, accumulate=True)
        assert _rel(acc, r0 + 1) < 1e-4
    set_sm_reserve(20)
    try:
        assert _rel(gemm(a, b, b_mn=True, out_fp32=True), r0) < 1e-4
    finally:
        set_sm_reserve(0)


def test_gemm_split_on_more_streams_than_workspaces():
    """The ninth stream takes the place of the first, which gets a new workspace when it comes back."""
    from pippy_b200.ops import gemm as mod

    a, b = _bf16(77, 4096), _bf16(4096, 4096)
    out = mod.gemm(a, b, b_mn=True)
    streams = [torch.cuda.Stream() for _ in range(mod._MAX_SPLIT_WS + 3)]
    torch.cuda.synchronize()
    results = []
    for _ in range(3):
        for s in streams:
            with torch.cuda.stream(s):
                results.append(mod.gemm(a, b, b_mn=True))
    torch.cuda.synchronize()
    assert len(mod._SPLIT_WS) <= mod._MAX_SPLIT_WS
    assert all(torch.equal(out, r) for r in results)


@pytest.mark.parametrize("M,N,K", [(77, 4096, 4096), (2048, 768, 16384)])
def test_gemm_split_ignores_leftover_counters(M, N, K):
    """Whatever a launch that gave up left in the arrival counters of the kept workspace, the next call is right."""
    from pippy_b200.ops import _lib
    from pippy_b200.ops import gemm as mod

    a, b = _bf16(M, K), _bf16(K, N)
    out = mod.gemm(a, b, b_mn=True)
    ws = mod._SPLIT_WS[(a.device.index, _lib.stream_addr())]
    counters = ws[-mod._COUNTER_BYTES:].view(torch.int64)
    used = counters.clone()
    assert used.any()
    for left in (torch.ones_like(used), used, used - 1, torch.randint(-2 ** 62, 2 ** 62, used.shape, device="cuda")):
        counters.copy_(left)
        for _ in range(2):
            assert torch.equal(mod.gemm(a, b, b_mn=True), out)


def test_gemm_without_memory_for_a_split(monkeypatch):
    """A call whose workspace cannot be allocated runs unsplit, keeps nothing, and the next one tries again."""
    from pippy_b200.ops import gemm as mod

    def refuse(device):
        raise torch.OutOfMemoryError("no memory left")

    a, b = _bf16(77, 4096), _bf16(4096, 4096)
    split = mod.gemm(a, b, b_mn=True)
    monkeypatch.setattr(mod, "_SPLIT_WS", type(mod._SPLIT_WS)())
    with monkeypatch.context() as m:
        m.setattr(mod, "_new_split_ws", refuse)
        whole = mod.gemm(a, b, b_mn=True)
        assert _rel(whole, a.float() @ b.float()) < 1e-2 and not mod._SPLIT_WS
    assert torch.equal(mod.gemm(a, b, b_mn=True), split) and len(mod._SPLIT_WS) == 1


@pytest.mark.parametrize("H", [768, 4096, 5120])
@pytest.mark.parametrize("layer", [False, True])
def test_norm(H, layer):
    from pippy_b200.ops import functional as pf

    T = 515
    x = _bf16(T, H).requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_()
    b = (0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_() if layer else None
    dy = _bf16(T, H)
    y = pf.layer_norm(x, w, b, 1e-5) if layer else pf.rms_norm(x, w, 1e-5)
    y.backward(dy)
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    if layer:
        bf = b.detach().float().requires_grad_()
        yr = F.layer_norm(xf, (H,), wf, bf, 1e-5)
    else:
        yr = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    yr.backward(dy.float())
    assert _rel(y, yr) < 1e-2
    assert _rel(x.grad, xf.grad) < 1e-2
    assert _rel(w.grad, wf.grad) < 2e-2
    if layer:
        assert _rel(b.grad, bf.grad) < 2e-2


def test_norm_fork_adds_the_residual_gradient():
    """``rms_norm_fork`` hands back its input for the residual branch; the gradient that returns through it is added
    to the norm's input gradient by the backward kernel."""
    from pippy_b200.ops import functional as pf

    T, H = 515, 4096
    x = _bf16(T, H).requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_()
    dy, dr = _bf16(T, H), _bf16(T, H)
    y, xr = pf.rms_norm_fork(x, w, 1e-5)
    assert xr.data_ptr() == x.data_ptr()
    torch.autograd.backward([y, xr], [dy, dr])
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    torch.autograd.backward([yr, xf * 1.0], [dy.float(), dr.float()])
    assert _rel(y, yr) < 1e-2
    assert _rel(x.grad, xf.grad) < 1e-2
    assert _rel(w.grad, wf.grad) < 2e-2
    # only the residual branch used: the gradient passes through
    x2 = _bf16(T, H).requires_grad_()
    _, xr2 = pf.rms_norm_fork(x2, w, 1e-5)
    xr2.backward(dr)
    assert torch.equal(x2.grad, dr)


def test_llama_block_matches_fp32_reference():
    """One decoder layer on the kernels (bf16) against the same layer's plain PyTorch path in fp32 on the CPU:
    output, input gradient and the gradients of both norm weights and of the down projection."""
    from pippy_b200.models.llama import LlamaBlock, LlamaConfig

    cfg = LlamaConfig(vocab_size=256, dim=512, n_layers=1, n_heads=4, ffn_dim=1024)
    B, S = 2, 128
    torch.manual_seed(3)
    ref = LlamaBlock(cfg, dtype=torch.float32)
    with torch.no_grad():
        for name, prm in ref.named_parameters():
            if name.endswith("norm.weight"):
                prm.add_(0.1 * torch.randn_like(prm))
            prm.copy_(prm.bfloat16().float())  # both sides start from the same bf16-representable weights
    blk = LlamaBlock(cfg, device="cuda", dtype=torch.bfloat16)
    blk.load_state_dict({k: v.bfloat16() for k, v in ref.state_dict().items()})
    x = (0.5 * torch.randn(B * S, cfg.dim)).bfloat16()
    dy = (0.1 * torch.randn(B * S, cfg.dim)).bfloat16()
    xg = x.cuda().requires_grad_()
    out = blk(xg, B, S)
    out.backward(dy.cuda())
    xr = x.float().requires_grad_()
    out_ref = ref(xr, B, S)
    out_ref.backward(dy.float())
    assert _rel(out.cpu(), out_ref) < 2e-2
    assert _rel(xg.grad.cpu(), xr.grad) < 3e-2
    got = dict(blk.named_parameters())
    for name in ("attention_norm.weight", "ffn_norm.weight", "feed_forward.w_down.weight"):
        want = dict(ref.named_parameters())[name].grad
        g = got[name].grad if got[name].grad is not None else got[name].main_grad
        assert _rel(g.cpu(), want) < 5e-2, name


def test_swiglu_and_gelu_linear():
    from pippy_b200.ops import functional as pf

    T, Fd = 300, 1408
    gu = _bf16(T, 2 * Fd).requires_grad_()
    d = _bf16(T, Fd)
    out = pf.swiglu(gu)
    out.backward(d)
    gf = gu.detach().float().requires_grad_()
    g, u = gf.chunk(2, -1)
    ref = F.silu(g) * u
    ref.backward(d.float())
    assert _rel(out, ref) < 1e-2 and _rel(gu.grad, gf.grad) < 1e-2

    x = _bf16(T, 256).requires_grad_()
    w = _bf16(512, 256, scale=0.05).requires_grad_()
    bias = _bf16(512, scale=0.1).requires_grad_()
    res = _bf16(T, 512).requires_grad_()
    dy = _bf16(T, 512)
    y = pf.linear(x, w, bias, residual=res, activation="gelu_tanh")
    y.backward(dy)
    xf, wf, bf, rf = (t.detach().float().requires_grad_() for t in (x, w, bias, res))
    yr = F.gelu(F.linear(xf, wf, bf), approximate="tanh") + rf
    yr.backward(dy.float())
    assert _rel(y, yr) < 1e-2
    assert _rel(x.grad, xf.grad) < 2e-2
    assert _rel(w.grad, wf.grad) < 2e-2
    assert _rel(bias.grad, bf.grad) < 2e-2
    assert _rel(res.grad, rf.grad) < 1e-2


def test_linear_main_grad_accumulates_fp32():
    from pippy_b200.ops import functional as pf

    x = _bf16(256, 128).requires_grad_()
    w = _bf16(384, 128, scale=0.05).requires_grad_()
    w.main_grad = torch.zeros(384, 128, device="cuda")
    for _ in range(2):
        pf.linear(x, w).backward(torch.ones(256, 384, device="cuda", dtype=torch.bfloat16))
    ref = 2 * torch.ones(256, 384, device="cuda").t() @ x.detach().float()
    assert w.grad is None and _rel(w.main_grad, ref) < 1e-3


@pytest.mark.parametrize("T,C,ld", [(1, 8, 8), (33, 264, 272), (2048, 768, 768), (1000, 2304, 2304), (257, 1024, 1028), (100, 30, 30),
                                    (2048, 3072, 3072), (5003, 2304, 2304), (9001, 776, 784)])
def test_column_sums(T, C, ld):
    """Bias gradients: whole and partial 256-column groups, fewer rows than a CTA takes, several trips of a CTA's row loop
    (the last three), pitches that are no multiple of 8 (the 4-byte kernel).  fp32 sums of T bf16 values: the order changes them by T * 2^-24 of the absolute sum at most."""
    from pippy_b200.ops import _lib

    x = _bf16(T, ld)
    out = torch.ones(C, device="cuda")
    _lib.check(_lib.lib().pb_colsum_bf16(_lib.ptr(x), _lib.ptr(out), _lib.c_ll(T), _lib.c_int(C), _lib.c_ll(ld),
                                         _lib.stream_ptr()), "pb_colsum_bf16")
    ref = x[:, :C].double().sum(0) + 1
    bound = (T + 8) * 2 ** -24 * (x[:, :C].double().abs().sum(0) + 1)
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("T", [1, 31, 33, 257, 3000])
@pytest.mark.parametrize("layer", [False, True])
def test_norm_weight_gradient_fold(T, layer):
    """From one partial row to a full grid of them, against fp64; the bias has its own half of the fold."""
    from pippy_b200.ops import functional as pf

    H = 776
    x = _bf16(T, H).requires_grad_()
    w, b = torch.nn.Parameter(_bf16(H)), torch.nn.Parameter(_bf16(H))
    w.main_grad, b.main_grad = (torch.randn(H, device="cuda") for _ in range(2))
    w0, b0 = w.main_grad.double(), b.main_grad.double()
    dy = _bf16(T, H)
    (pf.layer_norm(x, w, b) if layer else pf.rms_norm(x, w)).backward(dy)
    xd = x.detach().double()
    mean = xd.mean(-1, keepdim=True) if layer else 0.0
    xh = (xd - mean) * torch.rsqrt((xd - mean).pow(2).mean(-1, keepdim=True) + 1e-5)
    terms = dy.double() * xh
    assert ((w.main_grad.double() - w0 - terms.sum(0)).abs() <= 1e-5 * (terms.abs().sum(0) + 1)).all()
    if layer:
        assert ((b.main_grad.double() - b0 - dy.double().sum(0)).abs() <= 1e-5 * (dy.double().abs().sum(0) + 1)).all()


def test_norm_backward_beside_other_streams_and_replays():
    """Weight gradients of the same width from two streams at once, and from a captured backward that is replayed beside
    eager ones: each has its own partial sums."""
    from pippy_b200.ops import functional as pf

    T, H = 2048, 1024
    x, dy = [_bf16(T, H).requires_grad_() for _ in range(2)], [_bf16(T, H) for _ in range(2)]
    ws = [torch.nn.Parameter(_bf16(H)) for _ in range(2)]
    for w in ws:
        w.main_grad = torch.zeros(H, device="cuda")

    def backward(i):
        return torch.autograd.grad(pf.rms_norm(x[i], ws[i]), x[i], dy[i])[0]

    refs = []
    for i in range(2):
        backward(i)
        refs.append(ws[i].main_grad.clone())
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        ws[0].main_grad.zero_()
        backward(0)
    for first in (lambda: (ws[0].main_grad.zero_(), backward(0)), graph.replay):
        for _ in range(20):
            with torch.cuda.stream(streams[0]):
                first()
            with torch.cuda.stream(streams[1]):
                ws[1].main_grad.zero_()
                backward(1)
            torch.cuda.synchronize()
            assert torch.equal(ws[0].main_grad, refs[0]) and torch.equal(ws[1].main_grad, refs[1])


def test_cross_entropy():
    from pippy_b200.ops import functional as pf

    T, V, Vp = 257, 1000, 1024
    logits = _bf16(T, Vp, scale=2.0).requires_grad_()
    tgt = torch.randint(0, V, (T,), device="cuda")
    tgt[5] = -100
    loss = pf.cross_entropy(logits, tgt, vocab_size=V, reduction="mean")
    (loss * 3.0).backward()
    lf = logits.detach().float().requires_grad_()
    ref = F.cross_entropy(lf[:, :V], tgt, reduction="mean", ignore_index=-100)
    (ref * 3.0).backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * abs(ref.item())
    assert (logits.grad.float() - lf.grad).abs().max().item() < 2e-4
    assert logits.grad[:, V:].abs().max().item() == 0


@pytest.mark.parametrize("V,pad", [(8, 0), (13, 3), (4096, 0), (4097, 7), (32000, 0), (50257, 47), (56000, 8), (56001, 7)])
@pytest.mark.parametrize("reduction", ["mean", "sum"])
def test_cross_entropy_class_counts(V, pad, reduction):
    """Around the class counts at which another kernel takes the row (4096, 56000) and around whole 16-byte vectors:
    loss, gradient (with an incoming gradient of 1 and of 3), ignored rows, columns at and beyond the padding, and the
    loss alone without a gradient."""
    from pippy_b200.ops import functional as pf

    T = 37
    logits = _bf16(T, V + pad, scale=3.0)
    logits[:, V:] = 1e4  # padding has to have no influence
    tgt = torch.randint(0, V, (T,), device="cuda")
    tgt[3], tgt[4], tgt[0] = -100, V - 1, 0
    lf = logits[:, :V].double().requires_grad_()
    ref = F.cross_entropy(lf, tgt, reduction=reduction, ignore_index=-100)
    ref.backward()
    for factor in (1.0, 3.0):
        x = logits.clone().requires_grad_()
        loss = pf.cross_entropy(x, tgt, vocab_size=V, reduction=reduction)
        assert abs(loss.item() - ref.item()) < 1e-5 * abs(ref.item())
        (loss * factor).backward()
        # one rounding to bf16 (relative 2^-8 at most), a second one with a factor, and 1e-4 for fp32 exponentials
        bound = (2 ** -8 if factor == 1.0 else 2 ** -7) + 1e-4
        assert ((x.grad[:, :V].double() - factor * lf.grad).abs() <= bound * factor * lf.grad.abs() + 1e-9).all()
        assert x.grad[3].abs().max().item() == 0 and (pad == 0 or x.grad[:, V:].abs().max().item() == 0)
    keep = logits.clone()
    with torch.no_grad():
        assert torch.equal(pf.cross_entropy(logits, tgt, vocab_size=V, reduction=reduction), loss.detach())
        assert torch.equal(logits, keep)
        pf.cross_entropy(logits, tgt, vocab_size=V, reduction=reduction, inplace=True)
        assert ((logits[:, :V].double() - lf.grad).abs() <= (2 ** -8 + 1e-4) * lf.grad.abs() + 1e-9).all()


@pytest.mark.parametrize("V", [1000, 32000, 60000])
def test_cross_entropy_infinite_and_nan_logits(V):
    """Masked classes (-inf, among them whole vectors at the start and a lone finite class), the type's lowest value, +inf
    and NaN in all three kernels, against 64 bits."""
    from pippy_b200.ops import functional as pf

    T, inf = 8, float("inf")
    logits = _bf16(T, V, scale=3.0)
    tgt = torch.randint(40, V, (T,), device="cuda")
    logits[0, :32] = -inf
    logits[1, :] = -inf
    logits[1, tgt[1]] = 2.0
    logits[2, 100:] = torch.finfo(torch.bfloat16).min
    tgt[2] = 50
    logits[3, tgt[3]] = -inf  # the loss is infinite, the gradient is not
    logits[4, 7] = inf
    logits[5, 9] = float("nan")
    logits[6, :] = -inf
    logits[7, ::2] = -inf
    tgt[7] = 41
    lf = logits.double().requires_grad_()
    rows = F.cross_entropy(lf, tgt, reduction="none")
    for i in range(T):
        x = logits[i : i + 1].clone().requires_grad_()
        loss = pf.cross_entropy(x, tgt[i : i + 1], reduction="sum")
        loss.backward()
        (grad,) = torch.autograd.grad(rows[i], lf, retain_graph=True)
        if rows[i].isnan():
            assert loss.isnan() and x.grad.isnan().any(), i
            continue
        assert loss.item() == rows[i].item() or abs(loss.item() - rows[i].item()) <= 1e-5 * abs(rows[i].item()) + 1e-5, i
        # one rounding to bf16 and 1e-4 for fp32 exponentials
        assert ((x.grad[0].double() - grad[i]).abs() <= (2 ** -8 + 1e-4) * grad[i].abs() + 1e-9).all(), i


def test_embedding():
    from pippy_b200.ops import functional as pf

    V, H, B, S = 500, 256, 3, 64
    wte = _bf16(V, H).requires_grad_()
    wpe = _bf16(S, H).requires_grad_()
    ids = torch.randint(0, V, (B, S), device="cuda")
    out = pf.embedding(ids, wte, wpe, S)
    d = _bf16(B * S, H)
    out.backward(d)
    wf, pf_ = wte.detach().float().requires_grad_(), wpe.detach().float().requires_grad_()
    pos = torch.arange(B * S, device="cuda") % S
    ref = F.embedding(ids.reshape(-1), wf) + F.embedding(pos, pf_)
    ref.backward(d.float())
    assert _rel(out, ref) < 1e-2
    assert _rel(wte.grad, wf.grad) < 1e-2 and _rel(wpe.grad, pf_.grad) < 1e-2


def test_fused_adamw_matches_torch():
    import torch.nn as nn

    from pippy_b200.optim import FlatParams, FusedAdamW

    ps = [nn.Parameter(_bf16(300, 70)), nn.Parameter(_bf16(129))]
    ref = [nn.Parameter(p.detach().float().clone()) for p in ps]
    flat = FlatParams(ps)
    opt = FusedAdamW(flat, lr=1e-2, weight_decay=0.1, master_weights=True)
    ropt = torch.optim.AdamW(ref, lr=1e-2, weight_decay=0.1)
    for _ in range(3):
        for p, r in zip(ps, ref):
            g = torch.randn_like(r)
            p.main_grad.copy_(g)
            r.grad = g.clone()
        opt.step(zero_grad=True)
        ropt.step()
    for p, r in zip(ps, ref):
        assert _rel(p, r) < 1e-2
        assert p.main_grad.abs().max().item() == 0
    assert _rel(opt.master[0][: ps[0].numel()].view_as(ref[0]), ref[0]) < 1e-5


def _attn_ref(q, k, v, causal, scale):
    # q [B,S,Hq,D], k/v [B,S,Hkv,D] fp32
    rep = q.shape[2] // k.shape[2]
    k = k.repeat_interleave(rep, dim=2)
    v = v.repeat_interleave(rep, dim=2)
    att = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    if causal:
        S = q.shape[1]
        att = att.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    return torch.einsum("bhqk,bkhd->bqhd", att.softmax(-1), v)


@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(2, 256, 4, 4, 128), (1, 384, 8, 2, 128), (2, 320, 4, 4, 64), (1, 1024, 2, 1, 64)])
def test_flash_attention_fwd_bwd(B, S, Hq, Hkv, D):
    from pippy_b200.ops import functional as pf

    T = B * S
    qkv = _bf16(T, (Hq + 2 * Hkv) * D).requires_grad_()
    do = _bf16(T, Hq * D)
    out = pf.rope_attention(qkv, None, None, B, S, Hq, Hkv, D)
    out.backward(do)
    qf = qkv.detach().float().requires_grad_()
    q = qf[:, : Hq * D].view(B, S, Hq, D)
    k = qf[:, Hq * D : (Hq + Hkv) * D].view(B, S, Hkv, D)
    v = qf[:, (Hq + Hkv) * D :].view(B, S, Hkv, D)
    ref = _attn_ref(q, k, v, True, 1 / math.sqrt(D)).reshape(T, Hq * D)
    ref.backward(do.float())
    assert _rel(out, ref) < 2e-2
    g, gr = qkv.grad.float(), qf.grad
    for name, sl in (("dq", slice(0, Hq * D)), ("dk", slice(Hq * D, (Hq + Hkv) * D)), ("dv", slice((Hq + Hkv) * D, None))):
        assert _rel(g[:, sl], gr[:, sl]) < 3e-2, name


def _check_attention(q, k, v, do, B, S, Hq, Hkv, D, causal, out, dq, dk, dv):
    """Every element of the output and of the gradients ([B * S, heads * D]) against 64 bits.  With u = 2^-8, twice the
    rounding of bf16 (the other half is for the fp32 work), P, dS and what is stored are off by u of themselves, and delta =
    dO . O inherits the error of the stored O.  Returns the scores."""
    scale, u, tiny = 1 / math.sqrt(D), 2.0 ** -8, 1e-30
    q, do = (t.double().view(B, S, Hq, D).transpose(1, 2) for t in (q, do))
    k, v = (t.double().view(B, S, Hkv, D).transpose(1, 2).repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    att = q @ k.transpose(2, 3) * scale
    if causal:
        att = att.masked_fill(torch.ones(S, S, device=q.device, dtype=torch.bool).triu(1), float("-inf"))
    p = att.softmax(-1)
    o = p @ v
    o_off = u * (p @ v.abs() + o.abs())
    dp = do @ v.transpose(2, 3) - (do * o).sum(-1, keepdim=True)
    ds = p * dp * scale
    ds_off = p * (u * dp.abs() + (do.abs() * o_off).sum(-1, keepdim=True)) * scale
    ref = {"dq": (ds @ k, ds_off @ k.abs()),
           "dk": (ds.transpose(2, 3) @ q, ds_off.transpose(2, 3) @ q.abs()),
           "dv": (p.transpose(2, 3) @ do, u * (p.transpose(2, 3) @ do.abs()))}
    got = {"dq": dq, "dk": dk, "dv": dv}
    assert ((out.double().view(B, S, Hq, D).transpose(1, 2) - o).abs() <= o_off + tiny).all()
    for name, (r, off) in ref.items():
        heads = Hq if name == "dq" else Hkv
        r, off = (t.reshape(B, heads, Hq // heads, S, D).sum(2) for t in (r, off))
        g = got[name].double().view(B, S, heads, D).transpose(1, 2)
        assert ((g - r).abs() <= off + u * r.abs() + tiny).all(), name
    return att


@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal", [
    (1, 640, 50, 50, 128, True), (2, 257, 40, 10, 128, True), (3, 129, 27, 27, 64, True), (1, 1, 148, 37, 128, True),
    (1, 1153, 32, 8, 64, True), (2, 300, 40, 40, 128, False), (1, 128, 148, 148, 64, False), (2, 1000, 20, 20, 128, True),
])
def test_flash_attention_many_tiles(B, S, Hq, Hkv, D, causal):
    """Enough tiles for two query tiles per CTA (148 pairs or more), with second tiles that are empty, ragged or full,
    several groups of heads in the tile order, and keys that fill no block."""
    from pippy_b200.ops import functional as pf

    T = B * S
    qkv = _bf16(T, (Hq + 2 * Hkv) * D).requires_grad_()
    do = _bf16(T, Hq * D)
    out = pf.rope_attention(qkv, None, None, B, S, Hq, Hkv, D, causal=causal)
    out.backward(do)
    q, k, v = qkv.detach().split([Hq * D, Hkv * D, Hkv * D], 1)
    dq, dk, dv = qkv.grad.split([Hq * D, Hkv * D, Hkv * D], 1)
    _check_attention(q, k, v, do, B, S, Hq, Hkv, D, causal, out, dq, dk, dv)


@pytest.mark.parametrize("B,S,H,D", [(1, 640, 50, 128), (1, 1100, 30, 64), (2, 896, 20, 64), (1, 1100, 30, 128),
                                     (1, 640, 4, 128), (1, 1100, 3, 64)])
@pytest.mark.parametrize("causal", [True, False])
def test_flash_attention_growing_scores(B, S, H, D, causal):
    """Keys that grow along the sequence: rows' maxima move by more than 2^8 again and again, so that the output
    accumulated so far has to be rescaled in later blocks, in both tiles of a CTA (and, with few heads, in the kernel
    with one)."""
    from pippy_b200.ops import functional as pf

    T, scale, w = B * S, 1 / math.sqrt(D), H * D
    q, k, v, do = (_bf16(T, w) for _ in range(4))
    k = (k.float() * (1 + torch.arange(S, device="cuda").repeat(B).view(T, 1) / 64)).bfloat16()
    qkv = torch.cat([q, k, v], 1)
    parts = qkv[:, :w], qkv[:, w : 2 * w], qkv[:, 2 * w :]
    o, lse = pf.flash_forward(*parts, B, S, H, H, D, scale, causal)
    dq, dk, dv, _ = pf.flash_backward(do, *parts, o, lse, B, S, H, H, D, scale, causal)
    att = _check_attention(q, k, v, do, B, S, H, H, D, causal, o, dq, dk, dv)
    assert (lse.double() - torch.logsumexp(att, -1)).abs().max() < 1e-3  # fp32 of values up to 100: 8e-6 each
    # running maxima after each block of 128 keys: enough rows move by more than 2^8 after their first block
    seen = torch.stack([a.amax(-1) for a in att.split(128, -1)], -1).cummax(-1).values * math.log2(math.e)
    assert (seen[..., 1:] > seen[..., :-1] + 8).any(-1).float().mean() > 0.1


def test_rope_attention_with_rotary():
    from pippy_b200.ops import functional as pf

    B, S, Hq, Hkv, D = 2, 256, 4, 2, 128
    T = B * S
    base = _bf16(T, (Hq + 2 * Hkv) * D)
    cos, sin = pf.rope_tables(S, D, 10000.0, "cuda")
    qkv = base.clone().requires_grad_()
    do = _bf16(T, Hq * D)
    qkv_in = qkv * 1  # the op rotates its input in place; give it a private buffer
    out = pf.rope_attention(qkv_in, cos, sin, B, S, Hq, Hkv, D)
    out.backward(do)
    qf = base.float().requires_grad_()
    q = pf._rope_ref(qf[:, : Hq * D].view(B, S, Hq, D), cos, sin)
    k = pf._rope_ref(qf[:, Hq * D : (Hq + Hkv) * D].view(B, S, Hkv, D), cos, sin)
    v = qf[:, (Hq + Hkv) * D :].view(B, S, Hkv, D)
    ref = _attn_ref(q.float(), k.float(), v, True, 1 / math.sqrt(D)).reshape(T, Hq * D)
    ref.backward(do.float())
    assert _rel(out, ref) < 2e-2
    assert _rel(qkv.grad, qf.grad) < 3e-2



@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 1)])
def test_gemm_many_tiles_per_cta(variant, a_mn, b_mn):
    """4096 x 8192 has 512 tiles of 256 x 256 (2048 of 128 x 128): every persistent CTA works through several
    tiles, so the accumulator ping-pong in TMEM, the wrap of the shared-memory ring across tiles and the grouped
    rasterisation all run, as they do in a training step."""
    from pippy_b200.ops.gemm import gemm

    M, N, K = 4096, 8192, 1024
    a = _bf16(K, M) if a_mn else _bf16(M, K)
    b = _bf16(K, N) if b_mn else _bf16(N, K)
    ref = (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
    out = gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn), variant=variant)
    assert _rel(out, ref) < 1e-2
    # a dropped or doubled tile shows as an O(1) error somewhere; rounding alone stays far below this everywhere
    assert ((out.float() - ref).abs() / ref.abs().clamp(min=8.0)).max().item() < 5e-2


def test_gemm_many_tiles_with_reserved_sms():
    """The grid that leaves SMs free for communication kernels covers the same tiles."""
    from pippy_b200.ops.gemm import gemm, set_sm_reserve

    M, N, K = 4096, 4096, 512
    a, b = _bf16(M, K), _bf16(N, K)
    ref = a.float() @ b.float().t()
    try:
        set_sm_reserve(8)
        out = gemm(a, b)
    finally:
        set_sm_reserve(0)
    assert _rel(out, ref) < 1e-2


def test_flash_attention_long_sequence():
    """The training shape's sequence length: 32 key blocks per query block, head dim 128."""
    from pippy_b200.ops import functional as pf

    B, S, Hq, Hkv, D = 1, 4096, 2, 2, 128
    T = B * S
    qkv = _bf16(T, (Hq + 2 * Hkv) * D).requires_grad_()
    do = _bf16(T, Hq * D)
    out = pf.rope_attention(qkv * 1, None, None, B, S, Hq, Hkv, D)
    out.backward(do)
    qf = qkv.detach().float().requires_grad_()
    q = qf[:, : Hq * D].view(B, S, Hq, D)
    k = qf[:, Hq * D : (Hq + Hkv) * D].view(B, S, Hkv, D)
    v = qf[:, (Hq + Hkv) * D :].view(B, S, Hkv, D)
    ref = _attn_ref(q, k, v, True, 1 / math.sqrt(D)).reshape(T, Hq * D)
    ref.backward(do.float())
    assert _rel(out, ref) < 2e-2
    g, gr = qkv.grad.float(), qf.grad
    for name, sl in (("dq", slice(0, Hq * D)), ("dk", slice(Hq * D, (Hq + Hkv) * D)), ("dv", slice((Hq + Hkv) * D, None))):
        assert _rel(g[:, sl], gr[:, sl]) < 3e-2, name


def test_peer_wait_runs_out_and_reports():
    """Failure detection on the device: the all-reduce kernel is launched as rank 0 of 2 with a second flag block
    that nobody ever writes (both "ranks" are buffers of this one GPU) and a wait limit of a few milliseconds.
    The kernel must return by itself, the error word must say "peer wait ran out", and the next launch must work."""
    import ctypes

    from pippy_b200.ops import _lib

    lib = _lib.lib()
    lib.pb_set_peer_wait_ms.argtypes = [ctypes.c_double]
    n = 1 << 16
    grad = torch.randn(n, device="cuda")
    staging = [torch.zeros(n, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    flags = [torch.zeros(64, device="cuda", dtype=torch.int32) for _ in range(2)]
    counter = torch.zeros(2, device="cuda", dtype=torch.int32)
    stag = (ctypes.c_void_p * 2)(*[ctypes.c_void_p(t.data_ptr()) for t in staging])
    flg = (ctypes.POINTER(ctypes.c_int) * 2)(
        *[ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_int)) for t in flags])
    grid = ctypes.c_int(0)
    err = _lib.err_word(grad.device)
    try:
        lib.pb_set_peer_wait_ms(5.0)
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record()
        rc = lib.pb_dp_allreduce(_lib.ptr(grad), stag, flg, _lib.ptr(counter), _lib.ptr(err), _lib.c_ll(n),
                                 _lib.c_float(0.5), _lib.c_int(0), _lib.c_int(2), _lib.c_int(1), _lib.c_int(8),
                                 ctypes.byref(grid), _lib.stream_ptr())
        assert rc == 0
        t1.record()
        torch.cuda.synchronize()
        assert t0.elapsed_time(t1) < 1000.0  # gave up after milliseconds, not after the default 3 s
        with pytest.raises(_lib.KernelError, match="peer wait ran out"):
            _lib.check_device_errors()
    finally:
        lib.pb_set_peer_wait_ms(0.0)
    # the context is intact: the same kernel as a one-rank group completes and scales the gradients
    before = grad.clone()
    rc = lib.pb_dp_allreduce(_lib.ptr(grad), stag, flg, _lib.ptr(counter), _lib.ptr(err), _lib.c_ll(n),
                             _lib.c_float(0.5), _lib.c_int(0), _lib.c_int(1), _lib.c_int(2), _lib.c_int(8),
                             ctypes.byref(grid), _lib.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    _lib.check_device_errors()
    torch.testing.assert_close(grad, (before * 0.5).bfloat16().float())


@pytest.mark.parametrize("schedule", ["interleaved_1f1b", "zero_bubble"])
def test_llama_activation_checkpointing_same_gradients(schedule):
    """Recomputing each block's forward inside the backward gives the gradients of the plain run: the kernels are
    deterministic, so everything but the atomically accumulated sums (norm weights, embedding rows) is bit-equal."""
    from pippy_b200.models.llama import LlamaConfig
    from pippy_b200.train import build_llama_pipeline

    dev = torch.device("cuda", 0)
    cfg = LlamaConfig(vocab_size=1024, dim=512, n_layers=4, n_heads=4, ffn_dim=1024)
    ids = torch.randint(0, cfg.vocab_size, (4, 256), device=dev)
    grads, losses = {}, {}
    for ckpt in (False, True):
        pipe = build_llama_pipeline(cfg, 4, 256, 2, dev, schedule=schedule, virtual_stages=2, seed=11,
                                    with_optimizer=True, activation_checkpointing=ckpt)
        pipe.optimizer = None  # keep the accumulated gradients: compare them, not the updated weights
        losses[ckpt] = float(pipe.train_step(ids, ids))
        torch.cuda.synchronize()
        grads[ckpt] = {n: p.main_grad.clone() for st in pipe.stages for n, p in st.submod.named_parameters()}
    assert abs(losses[True] - losses[False]) < 1e-6
    for n, g in grads[False].items():
        assert g.abs().max().item() > 0, n
        assert _rel(grads[True][n], g) < 1e-3, n


def test_moe_router_kernels():
    """softmax / top-k / normalised weights / load-balance loss / positions, and the logit gradient, against the
    plain PyTorch statement."""
    from pippy_b200.parallel.ep import EPContext, _Plan, _RouteFn

    T, E, k, H = 1000, 8, 2, 64
    ep = EPContext(None, max_tokens=T, hidden=H, top_k=k, n_experts=E)
    logits = _bf16(T, E, scale=1.5).requires_grad_()
    plan = _Plan(ep, T)
    topw, aux = _RouteFn.apply(logits, plan, E, k)
    gw = torch.randn(T, k, device="cuda")
    ((topw * gw).sum() + 0.37 * aux).backward()

    lf = logits.detach().float().requires_grad_()
    probs = lf.softmax(-1)
    ri = torch.sort(probs, dim=-1, descending=True, stable=True).indices[:, :k]  # ties: lower index first
    rw = probs.gather(-1, ri)
    rwn = rw / rw.sum(-1, keepdim=True)
    share = torch.bincount(ri.reshape(-1), minlength=E).float() / (T * k)
    raux = E * (share * probs.mean(0)).sum()
    ((rwn * gw).sum() + 0.37 * raux).backward()
    assert torch.equal(plan.expert.view(T, k).long(), ri)
    torch.testing.assert_close(topw, rwn, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(aux, raux, rtol=1e-5, atol=1e-6)
    assert torch.equal(plan.counts.long(), torch.bincount(ri.reshape(-1), minlength=E))
    # positions: assignment (t, j) is the n-th token (in token order) that chose its expert
    flat = ri.reshape(-1)
    want = torch.empty_like(flat)
    for e in range(E):
        idx = (flat == e).nonzero(as_tuple=True)[0]
        want[idx] = torch.arange(idx.numel(), device="cuda")
    assert torch.equal(plan.slot.long(), want)
    assert _rel(logits.grad, lf.grad) < 1e-2


@pytest.mark.parametrize("T", [384, 1500])
def test_moe_layer_one_rank_against_dense(T):
    """The whole expert-parallel layer (route, dispatch, grouped GEMMs, combine and their backward) with an
    expert-parallel group of one rank, against the dense PyTorch statement of the layer."""
    from pippy_b200.parallel.ep import EPContext, MoEFeedForward

    H, Fd, E, k = 256, 512, 4, 2
    ep = EPContext(None, max_tokens=T, hidden=H, top_k=k, n_experts=E, capacity_factor=1.0)
    torch.manual_seed(5)
    dense = MoEFeedForward(H, Fd, E, k, None, 1, 0, aux_coef=0.01, device="cuda", dtype=torch.bfloat16)
    fused = MoEFeedForward(H, Fd, E, k, ep, 1, 0, aux_coef=0.01, device="cuda", dtype=torch.bfloat16)
    fused.load_state_dict(dense.state_dict())
    for it in range(2):  # the second pass reuses buffers and flags
        x = _bf16(T, H)
        dy = _bf16(T, H)
        xa, xb = x.clone().requires_grad_(), x.clone().requires_grad_()
        for m in (dense, fused):
            for p in m.parameters():
                p.grad = None
        out = fused(xa)
        out.backward(dy)
        ref = dense(xb)
        ref.backward(dy)
        torch.cuda.synchronize()
        assert _rel(out, ref) < 2e-2, ("out", it)
        assert _rel(xa.grad, xb.grad) < 2e-2, ("dx", it)
        assert _rel(fused.router.grad[:E], dense.router.grad[:E]) < 3e-2, ("drouter", it)
        assert _rel(fused.w_down.grad, dense.w_down.grad) < 2e-2, ("dWdown", it)
        assert _rel(fused.w_gate_up.grad, dense.w_gate_up.grad) < 2e-2, ("dWgu", it)
        assert abs(float(fused.last_aux_loss) - float(dense.last_aux_loss)) < 1e-3


def test_bounds_checking_library_reports_bad_indices():
    """The debug library (PIPPY_BOUNDS_CHECK=1) validates indices read from tensors: a token id and a class label
    outside their tables are reported through the device error word and the accesses are skipped, so the kernels
    finish, the context stays usable and the in-range rows are still right."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = """
import torch
from pippy_b200.ops import _lib, functional as pf
assert _lib.bounds_check_enabled()
_lib.err_word(torch.device("cuda", 0))
wte = torch.randn(100, 64, device="cuda").bfloat16()
ids = torch.tensor([[1, 5, 250, 7]], device="cuda")          # 250 is outside the 100-row table
out = pf.embedding(ids, wte)
torch.cuda.synchronize()
assert torch.equal(out[0], wte[1]) and torch.equal(out[3], wte[7])
try:
    _lib.check_device_errors()
    raise SystemExit("the bad token id was not reported")
except _lib.KernelError as e:
    assert "code 5" in str(e), e
logits = torch.randn(4, 104, device="cuda").bfloat16()
tgt = torch.tensor([3, 99, 1000, 5], device="cuda")           # 1000 is outside the 100 classes
loss = pf.cross_entropy(logits, tgt, vocab_size=100, reduction="sum")
torch.cuda.synchronize()
try:
    _lib.check_device_errors()
    raise SystemExit("the bad label was not reported")
except _lib.KernelError as e:
    assert "code 5" in str(e), e
ok = pf.cross_entropy(logits, torch.tensor([3, 99, 0, 5], device="cuda"), vocab_size=100, reduction="sum")
torch.cuda.synchronize()
_lib.check_device_errors()
print("bounds-check build ok", float(loss), float(ok))
"""
    env = dict(os.environ, PIPPY_BOUNDS_CHECK="1", PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-3000:]
    assert "bounds-check build ok" in res.stdout
