"""norm->linear / GLU->linear recompute blocks against the separate ops and an fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref_norm_linear(x, res, nw, w, eps):
    h = x.float() + (0 if res is None else res.float())
    h = h.to(torch.bfloat16).float()
    y = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + eps) * nw.float()
    return y.to(torch.bfloat16).float() @ w.float().t(), h


@pytest.mark.parametrize("with_res", [False, True])
def test_norm_linear_matches_reference(with_res):
    from trainscale_b200.ops import fused_blocks
    torch.manual_seed(0)
    T, H, N = 512, 1024, 768
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    res = torch.randn(T, H, device="cuda", dtype=torch.bfloat16, requires_grad=True) if with_res else None
    nw = (1 + 0.1 * torch.randn(H, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(N, H, device="cuda") / H ** 0.5).to(torch.bfloat16).requires_grad_(True)
    out, h = fused_blocks.norm_linear(x, res, nw, w, 1e-5)
    gout, gh = torch.randn_like(out), torch.randn_like(h)
    (out.float() * gout.float()).sum().backward(retain_graph=True) if not with_res else \
        ((out.float() * gout.float()).sum() + (h.float() * gh.float()).sum()).backward()
    xr, nwr, wr = (t.detach().float().requires_grad_(True) for t in (x, nw, w))
    rr = res.detach().float().requires_grad_(True) if with_res else None
    hr = xr + (0 if rr is None else rr)
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-5) * nwr
    outr = yr @ wr.t()
    loss = (outr * gout.float()).sum() + ((hr * gh.float()).sum() if with_res else 0)
    loss.backward()

    def close(a, b, tol=3e-2):
        return (a.float() - b).abs().max().item() <= tol * max(b.abs().max().item(), 1.0)

    assert close(out, outr)
    assert close(x.grad, xr.grad)
    assert close(nw.grad, nwr.grad, 5e-2)
    assert close(w.grad, wr.grad)
    if with_res:
        assert close(res.grad, rr.grad)


def test_glu_linear_matches_reference():
    from trainscale_b200.ops import fused_blocks
    torch.manual_seed(1)
    T, I, N = 384, 1024, 512
    gu = torch.randn(T, 2 * I, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(N, I, device="cuda") / I ** 0.5).to(torch.bfloat16).requires_grad_(True)
    out = fused_blocks.glu_linear(gu, w, "silu")
    go = torch.randn_like(out)
    out.backward(go)
    gur, wr = gu.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    g, u = gur.chunk(2, -1)
    outr = (torch.nn.functional.silu(g) * u) @ wr.t()
    outr.backward(go.float())
    for a, b in ((out, outr), (gu.grad, gur.grad), (w.grad, wr.grad)):
        assert (a.float() - b).abs().max().item() <= 3e-2 * max(b.abs().max().item(), 1.0)


def test_decoder_layer_op_selective_equals_plain_path():
    from trainscale_b200.models.llama import LlamaConfig, LlamaForCausalLM
    torch.manual_seed(2)
    cfg = LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, max_position_embeddings=256)
    m = LlamaForCausalLM(cfg).cuda().to(torch.bfloat16).train()
    ids = torch.randint(0, 512, (2, 128), device="cuda")
    loss0 = m(input_ids=ids, labels=ids).loss
    loss0.backward()
    g0 = {n: p.grad.clone() for n, p in m.named_parameters()}
    m.zero_grad(set_to_none=True)
    m.op_selective_recompute(True)
    loss1 = m(input_ids=ids, labels=ids).loss
    loss1.backward()
    assert abs(loss0.item() - loss1.item()) < 1e-3
    for n, p in m.named_parameters():
        d = (p.grad.float() - g0[n].float()).abs().max().item()
        assert d <= 2e-2 * max(g0[n].float().abs().max().item(), 1e-3), n


# one vector per row, rows whose vectors are no multiple of a block, both sides of the unrolled loop's remainder
@pytest.mark.parametrize("rows,I", [(1, 8), (3, 24), (257, 1376), (300, 2048)])
@pytest.mark.parametrize("act", [0, 1, 2])
def test_product_and_gradient_in_one_pass(rows, I, act):
    """The bits of the two separate kernels."""
    from trainscale_b200.ops import activation
    torch.manual_seed(0)
    gu, d = torch.randn(rows, 2 * I, device="cuda").bfloat16(), torch.randn(rows, I, device="cuda").bfloat16()
    dgu, g = activation.glu_bwd_both_raw(d, gu, act)
    assert torch.equal(g, activation.glu_fwd_raw(gu, act)) and torch.equal(dgu, activation.glu_bwd_raw(d, gu, act))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("first", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 4097, 1 << 20])
def test_squared_norm_of_any_alignment(dtype, first, n):
    """fp32 sums in some order: 2^-23 for each of the at most n / threads + log steps, here a generous 1e-5."""
    import ctypes
    from trainscale_b200.ops import _lib
    torch.manual_seed(0)
    x = torch.randn(n + first, device="cuda").to(dtype)[first:]
    out = torch.zeros(1, device="cuda")
    rc = _lib.load("elementwise").ts_sumsq(_lib.ptr(x), int(dtype == torch.bfloat16), ctypes.c_longlong(n), _lib.ptr(out), _lib.ptr(None),
                                           ctypes.c_float(0.5), _lib.stream_ptr())
    assert rc == 0
    ref = (x.double() * 0.5).square().sum()
    assert abs(float(out) - float(ref)) <= 1e-5 * float(ref)


# places per chunk of 32: one, a whole chunk and its neighbours, runs that cross one or many chunks, that begin or end on a border
@pytest.mark.parametrize("ids", [[3], [5] * 31 + [6], [1] * 32, [1] * 33, [2] * 16 + [4] * 40 + [7], [0] * 300, list(range(100)),
                                 [1] * 32 + [2] * 64 + [3] * 5, "random"])
@pytest.mark.parametrize("H", [8, 1032])
@pytest.mark.parametrize("added", [False, True])
def test_embedding_gradient_in_the_owners_rows(ids, H, added):
    """fp32 sums of bf16 rows: 2^-23 of the magnitudes for each term; rows of no token keep what they had."""
    from trainscale_b200.ops.embedding import TokenEmbedding
    torch.manual_seed(0)
    V = 400
    flat = torch.randint(0, V, (700,)) if ids == "random" else torch.tensor(ids)
    flat = flat[torch.randperm(len(flat))].cuda()
    emb = TokenEmbedding(V, H).to("cuda", torch.bfloat16)
    w, runs = emb.weight, []
    w._ts_unit = object()                              # as an engine's parameter has one
    dy = torch.randn(1, len(flat), H, device="cuda").bfloat16()
    before = torch.randn(V, H, device="cuda")
    for _ in range(2):
        w.main_grad, w.grad_added = before.clone(), added
        emb(flat.view(1, -1)).backward(dy)
        assert w.grad is None and w.grad_added
        runs.append(w.main_grad)
    assert torch.equal(*runs)
    base = before.double() if added else torch.zeros(V, H, device="cuda", dtype=torch.double)
    ref = base.index_add(0, flat, dy[0].double())
    size = base.abs().index_add(0, flat, dy[0].double().abs())
    assert ((runs[0].double() - ref).abs() <= 2.0 ** -23 * (len(flat) + 1) * size + 1e-30).all()
    del w.main_grad
    emb(flat.view(1, -1)).backward(dy)                 # without an owner: torch's own gradient
    assert w.grad is not None


def _owned_embedding(V=40, H=16):
    from trainscale_b200.ops.embedding import TokenEmbedding
    torch.manual_seed(0)
    emb = TokenEmbedding(V, H).to("cuda", torch.bfloat16)
    emb.weight._ts_unit, emb.weight.grad_added = object(), False
    emb.weight.main_grad = torch.full((V, H), 3.0, device="cuda")
    ids = torch.randint(0, V, (2, 9), device="cuda")
    return emb, ids, torch.randn(2, 9, H, device="cuda").bfloat16()


def _dense(emb, ids, dy):
    return torch.zeros_like(emb.weight.main_grad).index_add(0, ids.reshape(-1), dy.reshape(-1, dy.shape[-1]).float())


def test_embedding_weight_may_change_before_its_gradient():
    emb, ids, dy = _owned_embedding()
    y = emb(ids)
    with torch.no_grad():
        emb.weight.mul_(2)
    y.backward(dy)
    assert emb.weight.grad_added and torch.allclose(emb.weight.main_grad, _dense(emb, ids, dy), atol=1e-5)


@pytest.mark.parametrize("when", ["before", "between"])
@pytest.mark.parametrize("kind", ["register_hook", "register_post_accumulate_grad_hook"])
def test_hooks_see_the_embedding_gradient(when, kind):
    emb, ids, dy = _owned_embedding()
    seen, w = [], emb.weight
    hook = (lambda g: seen.append(g.clone())) if kind == "register_hook" else (lambda p: seen.append(p.grad.clone()))
    if when == "before":
        getattr(w, kind)(hook)
    y = emb(ids)
    if when == "between":
        getattr(w, kind)(hook)
    y.backward(dy)
    # the same gradient in bf16 (2^-8 of sums of a few unit values)
    assert len(seen) == 1 and torch.allclose(seen[0].float(), _dense(emb, ids, dy), atol=2e-2)
    assert torch.equal(w.grad, seen[0]) and not w.grad_added and (w.main_grad == 3.0).all()


def test_embedding_gradients_that_are_asked_for():
    """`torch.autograd.grad` returns the weight's gradient, once and again, and one of something else leaves the owner's alone."""
    emb, ids, dy = _owned_embedding()
    (g,) = torch.autograd.grad(emb(ids), emb.weight, dy)
    assert torch.allclose(g.float(), _dense(emb, ids, dy), atol=2e-2)
    scale = torch.ones((), device="cuda", requires_grad=True)
    torch.autograd.grad((emb(ids) * scale).float().sum(), scale)
    assert not emb.weight.grad_added and (emb.weight.main_grad == 3.0).all()
    # d/ds of sum(g * m), where g = s * (gradient for dy)
    (g,) = torch.autograd.grad(emb(ids) * scale, emb.weight, dy, create_graph=True)
    (d,) = torch.autograd.grad(g.float().sum(), scale)
    assert abs(float(d) - float(dy.float().sum())) <= 0.02 * float(dy.float().abs().sum())


def test_embedding_under_transforms():
    emb, ids, dy = _owned_embedding()
    want = torch.nn.functional.embedding(ids, emb.weight)
    assert torch.equal(torch.func.vmap(emb)(ids), want)
    t = torch.randn_like(emb.weight)
    with torch.autograd.forward_ad.dual_level():
        w = torch.autograd.forward_ad.make_dual(emb.weight, t)
        out = torch.func.functional_call(emb, {"weight": w}, (ids,))
        assert torch.equal(torch.autograd.forward_ad.unpack_dual(out).tangent, t[ids])
