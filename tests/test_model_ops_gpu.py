"""Fused model kernels (forward and backward) against PyTorch autograd in fp32."""
import pytest
import torch
import torch.nn.functional as tF

from dion_b200.models import functional as Fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rms_norm(dtype):
    torch.manual_seed(0)
    x = torch.randn(4, 37, 768, device="cuda").to(dtype).requires_grad_()
    xr = x.detach().float().requires_grad_()
    y = Fn.rms_norm(x)
    yr = tF.rms_norm(xr, (768,), eps=torch.finfo(dtype).eps)
    g = torch.randn_like(yr)
    y.backward(g.to(y.dtype))
    yr.backward(g)
    tol = 1e-5 if dtype == torch.float32 else 3e-2
    assert (y.float() - yr).abs().max().item() < tol
    assert (x.grad.float() - xr.grad).abs().max().item() < tol


def test_rms_norm_autocast_emits_bf16():
    x = torch.randn(8, 768, device="cuda", requires_grad=True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = Fn.rms_norm(x)
    assert y.dtype == torch.bfloat16
    y.float().sum().backward()
    assert x.grad.dtype == torch.float32


@pytest.mark.parametrize("D", [64, 128])
def test_rope_qknorm(D):
    torch.manual_seed(0)
    B, T, H = 2, 50, 6
    q = torch.randn(B, T, H, D, device="cuda").bfloat16().requires_grad_()
    k = torch.randn(B, T, H, D, device="cuda").bfloat16().requires_grad_()
    inv = 1.0 / (10000 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    fr = torch.outer(torch.arange(T, device="cuda").float(), inv)
    cos, sin = fr.cos().bfloat16(), fr.sin().bfloat16()
    qo, ko = Fn.rope_qknorm(q, k, cos, sin)
    qr, kr = q.detach().float().requires_grad_(), k.detach().float().requires_grad_()

    def ref(x):
        d = D // 2
        c, s = cos.float()[None, :, None, :], sin.float()[None, :, None, :]
        y = torch.cat([x[..., :d] * c + x[..., d:] * s, x[..., d:] * c - x[..., :d] * s], 3)
        return tF.rms_norm(y, (D,), eps=torch.finfo(torch.bfloat16).eps)

    qro, kro = ref(qr), ref(kr)
    gq, gk = torch.randn_like(qro), torch.randn_like(kro)
    (qo.float() * gq + ko.float() * gk).sum().backward()
    (qro * gq + kro * gk).sum().backward()
    assert (qo.float() - qro).abs().max().item() < 3e-2
    assert (ko.float() - kro).abs().max().item() < 3e-2
    assert (q.grad.float() - qr.grad).abs().max().item() < 5e-2
    assert (k.grad.float() - kr.grad).abs().max().item() < 5e-2


def test_qkv_rope_matches_unfused():
    """Fused projection + RoPE + QK-norm against the three separate linears in fp32."""
    torch.manual_seed(0)
    B, T, H, D = 2, 48, 4, 64
    C = H * D
    h = (torch.randn(B, T, C, device="cuda") * 0.5).bfloat16().requires_grad_()
    ws = [(torch.randn(C, C, device="cuda") * C ** -0.5).requires_grad_() for _ in range(3)]
    inv = 1.0 / (10000 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    fr = torch.outer(torch.arange(T, device="cuda").float(), inv)
    cos, sin = fr.cos().bfloat16(), fr.sin().bfloat16()
    q, k, v = Fn.qkv_rope(h, ws[0], ws[1], ws[2], cos, sin, H)
    assert q.shape == k.shape == v.shape == (B, T, H, D)
    gq, gk, gv = (torch.randn(B, T, H, D, device="cuda") for _ in range(3))
    (q.float() * gq + k.float() * gk + v.float() * gv).sum().backward()

    hr = h.detach().float().requires_grad_()
    wr = [w.detach().bfloat16().float().requires_grad_() for w in ws]

    def rope_norm(x):
        d = D // 2
        c, s = cos.float()[None, :, None, :], sin.float()[None, :, None, :]
        y = torch.cat([x[..., :d] * c + x[..., d:] * s, x[..., d:] * c - x[..., :d] * s], 3)
        return tF.rms_norm(y, (D,), eps=torch.finfo(torch.bfloat16).eps)

    qr = rope_norm((hr @ wr[0].T).view(B, T, H, D))
    kr = rope_norm((hr @ wr[1].T).view(B, T, H, D))
    vr = (hr @ wr[2].T).view(B, T, H, D)
    (qr * gq + kr * gk + vr * gv).sum().backward()
    for got, ref in ((q, qr), (k, kr), (v, vr)):
        assert (got.float() - ref).abs().max().item() < 5e-2
    assert (h.grad.float() - hr.grad).abs().max().item() < 0.05 * hr.grad.abs().max().item() + 5e-2
    for w, r in zip(ws, wr):
        assert w.grad.dtype == torch.float32
        assert (w.grad - r.grad).abs().max().item() < 0.03 * r.grad.abs().max().item() + 5e-2


def test_embedding_backward_matches_torch():
    torch.manual_seed(0)
    V, C = 1000, 64
    w = torch.randn(V, C, device="cuda", requires_grad=True)
    wr = w.detach().clone().requires_grad_()
    idx = torch.randint(0, 50, (4, 200), device="cuda")  # many repeated ids
    idx[0, 0] = V - 1
    g = torch.randn(4, 200, C, device="cuda")
    Fn.embedding(idx, w).backward(g)
    tF.embedding(idx, wr).backward(g)
    assert torch.allclose(w.grad, wr.grad, atol=1e-4, rtol=1e-5)
    assert w.grad[60:V - 1].abs().max().item() == 0.0


@pytest.mark.parametrize("T", [1, 64, 65, 640, 70001])
@pytest.mark.parametrize("C", [8, 264])
def test_embedding_backward_runs_across_chunks(T, C):
    """Skewed ids (neighbouring long runs), one id only, and a token count whose chunks are larger
    than 64 positions; fp32 sums of T terms in another order than the fp64 ones."""
    torch.manual_seed(1)
    V = 97
    g = torch.randn(T, C, device="cuda")
    w = torch.randn(V, C, device="cuda", requires_grad=True)
    u = torch.rand(T, device="cuda", dtype=torch.float64)
    for idx in ((V ** u).long().sub_(1).clamp_(0, V - 1), torch.full((T,), V - 1, device="cuda")):
        (gw,) = torch.autograd.grad(Fn.embedding(idx, w), w, g)
        ref = torch.zeros(V, C, device="cuda", dtype=torch.float64).index_add_(0, idx, g.double())
        mass = torch.zeros(V, C, device="cuda", dtype=torch.float64).index_add_(
            0, idx, g.double().abs())
        # each sum has at most T roundings of 2^-24 of a partial sum; far fewer in a tree of chunks
        assert ((gw.double() - ref).abs() <= 2.0 ** -24 * 1100 * mass + 1e-30).all()


def test_embedding_backward_long_runs_and_absent_rows():
    """Ids that occur hundreds of times (split over the block's warps), ids that occur once,
    rows that never occur (written as zeros, not left as allocated), a row count that is no
    multiple of the warps per block, and bit-identical results from call to call."""
    torch.manual_seed(3)
    V, C, T = 1003, 768, 4096
    w = torch.randn(V, C, device="cuda", requires_grad=True)
    idx = torch.randint(0, V, (T,), device="cuda")
    idx[:900] = 7            # one long run
    idx[900:1500] = V - 1    # another, in the last (partial) group of rows
    idx[1500:1565] = 500     # just above the threshold
    idx[1565:1629] = 501     # exactly at it
    idx = idx[torch.randperm(T, device="cuda")].reshape(4, T // 4)
    g = torch.randn(4, T // 4, C, device="cuda")
    junk = torch.full((V, C), float("nan"), device="cuda")   # what an uninitialised buffer may hold
    del junk
    (g1,) = torch.autograd.grad(Fn.embedding(idx, w), w, g)
    (g2,) = torch.autograd.grad(Fn.embedding(idx, w), w, g)
    assert torch.equal(g1, g2)
    ref = torch.zeros(V, C, device="cuda", dtype=torch.float64)
    ref.index_add_(0, idx.reshape(-1), g.reshape(-1, C).double())
    assert torch.isfinite(g1).all()
    assert (g1.double() - ref).abs().max().item() < 1e-3
    absent = torch.ones(V, dtype=torch.bool, device="cuda")
    absent[idx.reshape(-1)] = False
    assert absent.any() and g1[absent].abs().max().item() == 0.0


def test_linear_bf16_fp32_weight_grad():
    torch.manual_seed(0)
    x = torch.randn(3, 40, 256, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(128, 256, device="cuda") * 0.05).requires_grad_()
    y = Fn.linear(x, w)
    assert y.dtype == torch.bfloat16 and y.shape == (3, 40, 128)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().bfloat16().float().requires_grad_()
    yr = xr @ wr.T
    yr.backward(g.float())
    assert w.grad.dtype == torch.float32
    assert (y.float() - yr).abs().max().item() < 5e-2
    assert (w.grad - wr.grad).abs().max().item() < 1e-2 * wr.grad.abs().max().item() + 1e-3
    assert (x.grad.float() - xr.grad).abs().max().item() < 5e-2


def test_mlp_relu2_fused_matches_composition(monkeypatch):
    monkeypatch.setenv("DION_B200_FUSED_MLP", "1")
    torch.manual_seed(0)
    B, T, C = 2, 300, 256
    h = (torch.randn(B, T, C, device="cuda") * 0.5).bfloat16().requires_grad_()
    wfc = (torch.randn(4 * C, C, device="cuda") * C ** -0.5).requires_grad_()
    wpr = (torch.randn(C, 4 * C, device="cuda") * (4 * C) ** -0.5).requires_grad_()
    y = Fn.mlp_relu2(h, wfc, wpr)
    g = torch.randn_like(y)
    y.backward(g)
    hr = h.detach().float().requires_grad_()
    wf = wfc.detach().bfloat16().float().requires_grad_()
    wp = wpr.detach().bfloat16().float().requires_grad_()
    yr = torch.relu(hr @ wf.T).square() @ wp.T
    yr.backward(g.float())

    def close(a, b, tol=3e-2):
        return (a.float() - b).abs().max().item() < tol * b.abs().max().item() + 1e-3

    assert close(y, yr)
    assert close(h.grad, hr.grad)
    assert wfc.grad.dtype == torch.float32 and close(wfc.grad, wf.grad)
    assert close(wpr.grad, wp.grad)


def test_relu2():
    x = torch.randn(16, 3072, device="cuda").bfloat16().requires_grad_()
    xr = x.detach().float().requires_grad_()
    y = Fn.relu2(x)
    yr = tF.relu(xr).square()
    g = torch.randn_like(yr)
    y.backward(g.bfloat16())
    yr.backward(g)
    assert (y.float() - yr).abs().max().item() < 0.1
    assert (x.grad.float() - xr.grad).abs().max().item() < 0.1


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [64, 50304])
def test_cross_entropy(dtype, V):
    torch.manual_seed(0)
    N = 300
    logits = (torch.randn(N, V, device="cuda") * 2).to(dtype)
    tgt = torch.randint(0, V, (N,), device="cuda")
    tgt[::7] = -1
    lr = logits.detach().float().requires_grad_()
    ref = tF.cross_entropy(lr, tgt, ignore_index=-1)
    ref.backward()
    lg = logits.clone().requires_grad_()
    loss = Fn.cross_entropy(lg, tgt, ignore_index=-1)
    (loss * 0.5).backward()
    assert abs(float(loss) - float(ref)) < (1e-4 if dtype == torch.float32 else 2e-2)
    tol = 1e-6 if dtype == torch.float32 else 2e-4
    assert (lg.grad.float() - 0.5 * lr.grad).abs().max().item() < tol


def test_gpt_forward_backward_matches_torch_path():
    from dion_b200.models.gpt import GPT, GPTConfig
    torch.manual_seed(0)
    cfg = GPTConfig(sequence_len=64, vocab_size=512, n_layer=2, n_head=2, n_embd=128)
    m = GPT(cfg).cuda()
    m.init_weights()
    x = torch.randint(0, 512, (3, 64), device="cuda")
    y = torch.randint(0, 512, (3, 64), device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = m(x, y)
    loss.backward()
    g_fused = [p.grad.clone() for p in m.parameters()]
    m.zero_grad()
    mc = GPT(cfg)
    mc.load_state_dict({k: v.cpu() for k, v in m.state_dict().items()})
    for mod in mc.modules():
        if hasattr(mod, "init_inv_freq"):
            mod.init_inv_freq()
    lc = mc(x.cpu(), y.cpu())
    lc.backward()
    assert abs(float(loss) - float(lc)) < 5e-2
    for g, p in zip(g_fused, mc.parameters()):
        denom = p.grad.abs().max().item() + 1e-6
        assert (g.cpu() - p.grad).abs().max().item() / denom < 0.1


@pytest.mark.parametrize("D", [768, 2048, 3072])
def test_add_rms_norm(D):
    torch.manual_seed(0)
    x = torch.randn(3, 21, D, device="cuda", requires_grad=True)
    d = torch.randn(3, 21, D, device="cuda").bfloat16().requires_grad_()
    xr = x.detach().clone().requires_grad_()
    dr = d.detach().float().requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        xn, h = Fn.add_rms_norm(x, d)
    assert xn.dtype == torch.float32 and h.dtype == torch.bfloat16
    xnr = xr + dr
    hr = tF.rms_norm(xnr, (D,), eps=torch.finfo(torch.float32).eps)
    g1, g2 = torch.randn_like(xnr), torch.randn_like(hr)
    (xn * g1).sum().backward(retain_graph=True)
    (h.float() * g2).sum().backward()
    ((xnr * g1).sum() + (hr * g2).sum()).backward()
    assert (xn - xnr).abs().max().item() < 1e-5
    assert (h.float() - hr).abs().max().item() < 3e-2
    assert (x.grad - xr.grad).abs().max().item() < 2e-2  # g2 passed through bf16 h
    assert (d.grad.float() - dr.grad).abs().max().item() < 5e-2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T,heads,dim", [(1, 1, 2, 64), (1, 37, 4, 64), (3, 128, 2, 128), (2, 300, 3, 32)])
def test_blocks_without_gradients_match_the_general_forward(B, T, heads, dim, dtype):
    """Row counts below, at and above a tile of both product kernels.  Both sides round every
    product to bf16 (2^-9 each, over two blocks); the fused relu^2 skips one of the roundings."""
    from dion_b200.models import inference
    from dion_b200.models.gpt import GPT, GPTConfig
    from dion_b200.ops import _backend
    torch.manual_seed(0)
    model = GPT(GPTConfig(sequence_len=T, vocab_size=512, n_layer=2, n_head=heads,
                          n_embd=heads * dim)).cuda()
    model.init_weights()
    model.transformer.h.to(dtype)
    ids = torch.randint(0, 512, (B, T), device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        ref = model(ids, ids, return_logits=True).detach()
        with torch.no_grad():
            _backend.reset_launch_count()
            got = model(ids, ids, return_logits=True)
            assert _backend.launch_count() >= 17
            last = model(ids, return_logits=True)
            seen = []
            hook = model.transformer.h[1].mlp.c_fc.register_forward_hook(lambda *a: seen.append(1))
            hooked = model(ids, ids, return_logits=True)
            hook.remove()
    assert seen
    for x in (got, hooked):
        assert ((x - ref).norm() / ref.norm()).item() < 2e-2
    assert ((last[:, 0] - ref[:, -1]).norm() / ref[:, -1].norm()).item() < 2e-2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T,heads,dim", [(1, 1, 12, 64), (2, 63, 3, 128), (1, 129, 8, 64), (3, 65, 10, 32),
                                           (1, 257, 5, 64), (2, 130, 8, 128), (5, 200, 2, 64)])
def test_stack_of_blocks_matches_the_general_forward(B, T, heads, dim, dtype):
    """One call for all blocks: rows and keys below, at and above their tiles, one to eight CTAs to a
    cluster, column tiles of both widths, every head dimension.  Both sides round every product to
    bf16 (2^-9 each, over three blocks)."""
    from dion_b200.models import inference
    from dion_b200.models.gpt import GPT, GPTConfig
    from dion_b200.ops import _backend, gemm
    torch.manual_seed(1)
    model = GPT(GPTConfig(sequence_len=T, vocab_size=515, n_layer=3, n_head=heads,
                          n_embd=heads * dim)).cuda()
    model.init_weights()
    model.transformer.h.to(dtype)
    assert inference._stack_fits(B * T, T, heads * dim, 4 * heads * dim, dim, 3)
    ids = torch.randint(0, 515, (B, T), device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        ref = model(ids, ids, return_logits=True).detach()
        with torch.no_grad():
            _backend.reset_launch_count()
            got = model(ids, ids, return_logits=True)
            assert _backend.launch_count() == 3 * 5 + 2
            again = model(ids, ids, return_logits=True)
            last = model(ids, return_logits=True)
    gemm.check_status()
    assert ((got - ref).norm() / ref.norm()).item() < 2e-2
    assert torch.equal(got, again)
    assert last.shape == (B, 1, 515)
    assert ((last[:, 0] - ref[:, -1]).norm() / ref[:, -1].norm()).item() < 2e-2


def test_stack_of_blocks_in_a_captured_graph_and_on_a_side_stream():
    """The launches, which may start before their predecessors end, keep their order in a graph and
    on another stream than the default one, and see weights changed just before."""
    from dion_b200.models.gpt import GPT, GPTConfig
    torch.manual_seed(2)
    model = GPT(GPTConfig(sequence_len=96, vocab_size=512, n_layer=4, n_head=6, n_embd=384)).cuda()
    model.init_weights()
    ids = torch.randint(0, 512, (1, 96), device="cuda")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        eager = model(ids, return_logits=True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = model(ids, return_logits=True)
        for _ in range(3):
            out.zero_()
            graph.replay()
            assert torch.equal(out, eager)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for p in model.transformer.h.parameters():
                p.mul_(0.5)
            halved = model(ids, return_logits=True)
        torch.cuda.current_stream().wait_stream(side)
        graph.replay()
        assert torch.equal(out, halved) and not torch.equal(out, eager)
        with torch.enable_grad():
            ref = model(ids, ids, return_logits=True)[:, -1:].detach()
    assert ((halved - ref).norm() / ref.norm()).item() < 2e-2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,C,V", [(1, 768, 1003), (2, 100, 7), (3, 1024, 65), (4, 4, 1), (4, 640, 2053)])
def test_next_token_logits(B, C, V, dtype):
    """Exact products of bf16 numbers summed in fp32, then rounded to bf16 like the layer's result."""
    from dion_b200.models import inference
    torch.manual_seed(V)
    head = torch.nn.Linear(C, V, bias=False, device="cuda", dtype=dtype)
    h = torch.randn(B, 3, C, device="cuda").bfloat16()
    got = inference.next_token_logits(head, h)
    ref = h[:, -1:].double() @ head.weight.bfloat16().double().mT
    assert got.shape == (B, 1, V) and got.dtype == torch.float32
    assert torch.equal(got, got.bfloat16().float())
    size = (h[:, -1:].double().abs() @ head.weight.bfloat16().double().abs().mT)
    assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-6 * size).all()
    assert inference.next_token_logits(torch.nn.Linear(C, V, device="cuda"), h) is None   # a bias
    assert inference.next_token_logits(head, h.expand(3, -1, -1, -1).reshape(-1, 3, C)[:5]) is None \
        if 3 * B >= 5 else True


def test_replaced_modules_take_the_general_forward():
    """A block, a linear layer or an embedding of another type may look nothing like the original:
    the path without gradients leaves such a model to the modules."""
    from dion_b200.models.gpt import GPT, GPTConfig

    class Twice(torch.nn.Module):
        def forward(self, x, h=None):
            return 2 * x, Fn.rms_norm(2 * x)

    class Scaled(torch.nn.Linear):
        def forward(self, x):
            return 0.5 * super().forward(x)

    torch.manual_seed(0)
    ids = torch.randint(0, 512, (2, 24), device="cuda")
    for change in (lambda m: m.transformer.h.__setitem__(0, Twice()),
                   lambda m: setattr(m.transformer.h[1].mlp, "c_fc", Scaled(128, 512, bias=False).cuda())):
        model = GPT(GPTConfig(sequence_len=24, vocab_size=512, n_layer=2, n_head=2, n_embd=128)).cuda()
        model.init_weights()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            plain = model(ids, ids, return_logits=True).detach()
            change(model)
            ref = model(ids, ids, return_logits=True).detach()
            assert not torch.equal(ref, plain)       # the replacement counts with gradients too
            with torch.no_grad():
                got = model(ids, ids, return_logits=True)
        assert torch.equal(got, ref)


def _small_gpt(**changes):
    from dion_b200.models.gpt import GPT, GPTConfig
    torch.manual_seed(0)
    model = GPT(GPTConfig(**{**dict(sequence_len=32, vocab_size=512, n_layer=2, n_head=2, n_embd=128),
                             **changes})).cuda()
    model.init_weights()
    return model, torch.randint(0, 512, (2, 24), device="cuda")


def _native(model, ids, dtype=torch.bfloat16, enabled=True):
    """What the path without gradients says to this call: its result, or None."""
    from dion_b200.models import gpt, inference
    with torch.no_grad(), torch.autocast("cuda", dtype=dtype, enabled=enabled):
        return inference.hidden_states(model, ids, gpt._FORWARDS)


def test_blocks_without_gradients_refuse_what_they_do_not_compute():
    """Other types, shapes and settings than the native blocks are written for go to the general
    forward, which gives a result for each of these."""
    from torch import nn

    from dion_b200.models import gpt, inference

    def layer(m):
        return m.transformer.h[1].attn.c_proj

    def biased(m):
        layer(m).bias = nn.Parameter(torch.zeros(128, device="cuda"))

    def global_hook(m):
        return nn.modules.module.register_module_forward_hook(lambda *a: None)

    model, ids = _small_gpt()
    assert _native(model, ids) is not None
    assert _native(model, ids, dtype=torch.float16) is None
    assert _native(model, ids, enabled=False) is None
    assert _native(model, ids.cpu()) is None
    assert _native(model, ids[0]) is None
    assert _native(model, ids[:, :0]) is None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert inference.hidden_states(model, ids, gpt._FORWARDS) is None
    for change in (
            biased,
            lambda m: m.transformer.h[0].to(torch.bfloat16),                # mixed weight types
            lambda m: m.transformer.h.to(torch.float16),
            lambda m: m.transformer.wte.to(torch.bfloat16),
            lambda m: setattr(layer(m), "weight", nn.Parameter(layer(m).weight.detach().t())),
            lambda m: m.transformer.h[0].mlp.register_forward_pre_hook(lambda *a: None),
            lambda m: m.transformer.wte.register_forward_hook(lambda *a: None),
            lambda m: setattr(m.transformer.h[1].attn, "n_head", 4),
            lambda m: setattr(m.transformer.h[1].mlp, "forward", lambda x: x),
            global_hook):
        model, ids = _small_gpt()
        handle = change(model)
        assert _native(model, ids) is None
        if change is global_hook:
            handle.remove()
    model, ids = _small_gpt(n_embd=96)                                       # heads of 48
    assert _native(model, ids) is None


def test_blocks_without_gradients_are_seen_by_tracers_and_transforms():
    """Whatever watches or transforms operators sees all of them: the general forward runs."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Pass(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Count(TorchDispatchMode):
        products = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            Count.products += "mm" in str(func)
            return func(*args, **(kwargs or {}))

    model, ids = _small_gpt()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        want = model(ids, ids, return_logits=True)
        with Count():
            got = model(ids, ids, return_logits=True)
        assert Count.products >= 9          # four products in each of two blocks, and the head
        assert ((got - want).norm() / want.norm()).item() < 2e-2
        with torch.autograd.forward_ad.dual_level():
            assert _native(model, ids) is None
        with Pass():
            assert _native(model, ids) is None
        seen = []
        torch.func.vmap(lambda t: seen.append(_native(model, ids)) or t)(torch.zeros(2, device="cuda"))
        assert seen == [None]


@pytest.mark.parametrize("name", ["Block", "CausalSelfAttention", "MLP", "Rotary"])
def test_replaced_forward_of_a_class_is_called(name, monkeypatch):
    """A ``forward`` put on the class (as instrumentation and adapters do) counts without gradients
    too."""
    from dion_b200.models import gpt
    cls = getattr(gpt, name)
    torch.manual_seed(0)
    ids = torch.randint(0, 512, (2, 24), device="cuda")
    model = gpt.GPT(gpt.GPTConfig(sequence_len=24, vocab_size=512, n_layer=2, n_head=2,
                                  n_embd=128)).cuda()
    model.init_weights()
    own, seen = cls.forward, []

    def forward(self, *args):
        seen.append(1)
        return own(self, *args)

    monkeypatch.setattr(cls, "forward", forward)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        ref = model(ids, ids, return_logits=True).detach()
        with torch.no_grad():
            seen.clear()
            got = model(ids, ids, return_logits=True)
    assert len(seen) == 2
    assert torch.equal(got, ref)


@pytest.mark.parametrize("width,rows,native", [(768, 4096, True), (2048, 2048, True),
                                               (2048, 4096, False), (3072, 512, True),
                                               (3072, 2048, False)])
def test_wide_models_with_many_rows_take_the_library_products(width, rows, native):
    """Both sides of the line up to which the path without gradients gains (not how fast they are)."""
    from dion_b200.models import gpt, inference
    with torch.device("cuda"):
        model = gpt.GPT(gpt.GPTConfig(sequence_len=512, vocab_size=64, n_layer=1,
                                      n_head=width // 128, n_embd=width))
    model.init_weights()
    ids = torch.zeros(rows // 512, 512, dtype=torch.long, device="cuda")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        assert (inference.hidden_states(model, ids, gpt._FORWARDS) is not None) == native
