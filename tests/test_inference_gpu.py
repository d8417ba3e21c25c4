import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_decode_attention_matches_reference():
    import ctypes
    from trainscale_b200.ops import _lib
    from trainscale_b200.ops.attention import attention_reference
    torch.manual_seed(0)
    dev = "cuda"
    lib = _lib.load("decode")
    n, Hq, Hkv, D, bs = 3, 8, 2, 128, 16
    lens = [5, 700, 1300]
    nb = sum(-(-l // bs) for l in lens) + 4
    kc = torch.randn(nb, bs, Hkv, D, device=dev, dtype=torch.bfloat16)
    vc = torch.randn(nb, bs, Hkv, D, device=dev, dtype=torch.bfloat16)
    perm = torch.randperm(nb).tolist()
    maxb = max(-(-l // bs) for l in lens)
    bt = torch.zeros(n, maxb, dtype=torch.int32)
    used = 0
    for i, l in enumerate(lens):
        k = -(-l // bs)
        bt[i, :k] = torch.tensor(perm[used:used + k], dtype=torch.int32)
        used += k
    bt = bt.to(dev)
    sl = torch.tensor(lens, dtype=torch.int32, device=dev)
    q = torch.randn(n, Hq * D, device=dev, dtype=torch.bfloat16)
    out = torch.empty_like(q)
    chunk = 512
    splits = -(-max(lens) // chunk)
    po = torch.empty(n, Hq, splits, D, device=dev)
    pl = torch.empty(n, Hq, splits, device=dev)
    rc = lib.ts_decode_attention(_lib.ptr(q), Hq * D, _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(bt), maxb, _lib.ptr(sl),
                                 _lib.ptr(out), Hq * D, _lib.ptr(po), _lib.ptr(pl), n, Hq, Hkv, D, bs, chunk, splits,
                                 ctypes.c_float(1 / math.sqrt(D)), _lib.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    for i, l in enumerate(lens):
        idx = bt[i, :-(-l // bs)].long()
        k = kc[idx].reshape(-1, Hkv, D)[:l].unsqueeze(0)
        v = vc[idx].reshape(-1, Hkv, D)[:l].unsqueeze(0)
        ref = attention_reference(q[i].view(1, 1, Hq, D), k, v, True).reshape(-1)
        assert (out[i].float() - ref.float()).abs().max().item() < 2e-2


def test_engine_on_gpu_matches_full_forward_logits():
    from trainscale_b200.inference import CacheConfig, EngineConfig, GenerationParams, SOTAInferenceEngine
    from trainscale_b200.models.llama import LlamaConfig, build_model
    cfg = LlamaConfig(vocab_size=300, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, head_dim=64)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=1)
    eng = SOTAInferenceEngine(EngineConfig(model="tiny", cache=CacheConfig(block_size=16, num_gpu_blocks=256,
                                                                            max_model_len=512)), model=model)
    prompts = ["the quick brown fox jumps over the lazy dog " * 3, "hello"]
    res = eng.generate(prompts, GenerationParams(max_tokens=16, temperature=0.0, ignore_eos=True)).unwrap()
    tok = eng.core.tokenizer
    for p, r in zip(prompts, res):
        assert len(r.token_ids) == 16
        # teacher-forced check: the full-context forward ranks each generated token (near) first
        ids = [tok.bos_token_id] + tok.encode_raw(p) + r.token_ids
        with torch.no_grad():
            logits = model(torch.tensor([ids], device="cuda")).logits[0].float()
        n0 = len(ids) - 16
        for j, t in enumerate(r.token_ids):
            row = logits[n0 - 1 + j]
            assert row[t] >= row.max() - 0.15, (j, row[t].item(), row.max().item())


def test_cuda_graph_decode_matches_eager_decode():
    """The decode loop replayed from CUDA graphs (padded batch, spare cache block for the padding rows) produces the
    tokens of the eager loop, for a batch whose size is not a power of two and that shrinks as requests finish."""
    from trainscale_b200.inference import CacheConfig, EngineConfig, GenerationParams, SOTAInferenceEngine
    from trainscale_b200.models.llama import LlamaConfig, build_model
    from trainscale_b200.ops import _lib
    cfg = LlamaConfig(vocab_size=300, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, head_dim=64)
    prompts = [[5, 9, 200, 31, 77, 12] * 5, [8, 8, 101], [250, 3, 3, 3, 19, 44, 60, 2, 91] * 12, [17] * 40, [4, 5]]
    lens = [24, 9, 30, 17, 12]

    def run(eager):
        model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=1)
        eng = SOTAInferenceEngine(EngineConfig(model="tiny", enforce_eager=eager,
                                               cache=CacheConfig(block_size=16, num_gpu_blocks=256, max_model_len=512)),
                                  model=model)
        reqs = [eng.core.add_request(p, GenerationParams(max_tokens=n, temperature=0.0, ignore_eos=True))
                for p, n in zip(prompts, lens)]
        while eng.core.has_unfinished():
            eng.core.step()
        return [r.output_ids for r in reqs], eng

    want, _ = run(True)
    got, eng = run(False)
    assert eng.core.runner.graph_replays > 20 and len(eng.core.runner.graphs) >= 2
    torch.cuda.synchronize()
    _lib.raise_on_any_device_error()
    agree = sum(g == w for g, w in zip(got, want))
    # identical kernels on identical inputs: the sequences must be the same (a near-tie may flip at most one of them)
    assert agree >= len(want) - 1, (got, want)
    for g, w in zip(got, want):
        assert g[:6] == w[:6]


# (keys before the portion, its tokens): tile edges (128 keys, 128 / 256 query rows) and their neighbours, the smallest portions
@pytest.mark.parametrize("Hq,Hkv,D", [(4, 2, 64), (4, 1, 128), (3, 3, 64)])
@pytest.mark.parametrize("parts", [[(1, 2), (0, 2)], [(126, 2), (127, 2), (0, 129), (1, 127)], [(255, 257), (640, 3), (3, 256)],
                                   [(1000, 300)]])
def test_portions_against_the_cache_match_fp64(Hq, Hkv, D, parts):
    """Gathered keys and the flash kernel with split weights: bf16 rounding of the result (2^-9, doubled) plus what weights of
    16 bits leave of values up to about five (2^-16 * 5)."""
    from trainscale_b200.ops import _lib, flash
    torch.manual_seed(1)
    dev, bs, kw = "cuda", 16, Hkv * D
    lens = [s + n for s, n in parts]
    blocks = [-(-n // bs) for n in lens]
    kc, vc = (torch.randn(sum(blocks) + 1, bs, Hkv, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    kc[-1] = vc[-1] = float("nan")              # a block that nobody holds must not be read
    order, table = torch.randperm(sum(blocks)), torch.full((len(parts), max(blocks)), sum(blocks), dtype=torch.int32)
    for i, part in enumerate(order.split(blocks)):
        table[i, :blocks[i]] = part
        tail = lens[i] % bs
        if tail:
            kc[part[-1], tail:] = vc[part[-1], tail:] = float("nan")
    table = table.to(dev)
    rows = [-(-n // 128) * 128 for n in lens]
    i32 = dict(dtype=torch.int32, device=dev)
    starts, lens_d = torch.tensor([sum(rows[:i]) for i in range(len(rows))], **i32), torch.tensor(lens, **i32)
    cu = [3]                                     # three rows of others come first
    for _, n in parts:
        cu.append(cu[-1] + n)
    q = torch.randn(cu[-1], Hq * D + 2 * kw, device=dev, dtype=torch.bfloat16)
    out = torch.full((cu[-1], Hq * D), 7.0, device=dev, dtype=torch.bfloat16)
    kv = torch.full((sum(rows), 2 * kw), float("nan"), device=dev, dtype=torch.bfloat16)
    lib = _lib.load("decode")
    _lib.check(lib.ts_kv_gather(_lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), table.shape[1], _lib.ptr(starts), _lib.ptr(lens_d),
                                len(parts), max(lens), bs, kw, _lib.ptr(kv), _lib.stream_ptr()), "ts_kv_gather")
    flash.flash_portions(q, kv[:, :kw], kv[:, kw:], out, Hq, Hkv, D, torch.tensor(cu, **i32), starts, lens_d,
                         max(n for _, n in parts), 1 / math.sqrt(D))
    torch.cuda.synchronize()
    _lib.raise_on_any_device_error()
    assert (out[:3] == 7.0).all()
    for i, (s, n) in enumerate(parts):
        k, v = (c[table[i, :blocks[i]].long()].reshape(-1, Hkv, D)[:lens[i]].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        sc = torch.einsum("qhd,khd->hqk", q[cu[i]:cu[i + 1], :Hq * D].double().view(n, Hq, D), k) / math.sqrt(D)
        hidden = torch.arange(lens[i], device=dev) > torch.arange(s, s + n, device=dev).unsqueeze(1)
        ref = torch.einsum("hqk,khd->qhd", torch.softmax(sc.masked_fill(hidden, float("-inf")), -1), v).reshape(n, -1)
        err = (out[cu[i]:cu[i + 1]].double() - ref).abs()
        assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -16 * 5).all(), float(err.max())


def test_mixed_steps_give_the_logits_of_the_whole_sequence():
    """Decoding rows beside first and further portions of prompts in one step; groups of sequences that are gathered apart."""
    from trainscale_b200.inference import engine as E
    from trainscale_b200.inference.batch import StepEntry
    from trainscale_b200.models.llama import LlamaConfig, build_model
    cfg = LlamaConfig(vocab_size=300, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, head_dim=64)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=1)
    config = E.EngineConfig(model="tiny", cache=E.CacheConfig(block_size=16, num_gpu_blocks=256, max_model_len=1024))
    core = E.EngineCore(config, model=model)
    g = torch.Generator().manual_seed(3)
    ids = {s: torch.randint(0, 300, (n,), generator=g).tolist() for s, n in ((0, 9), (1, 400), (2, 150), (3, 33))}
    want = {s: model(torch.tensor([t], device="cuda")).logits[0].float().detach() for s, t in ids.items()}
    limit, E.GATHER_ROWS = E.GATHER_ROWS, 256
    try:
        at = {s: 0 for s in ids}
        for step in ([(0, 7), (1, 130)], [(2, 1), (1, 200), (0, 1), (3, 20)], [(3, 13), (2, 149), (1, 70), (0, 1)]):
            logits = core.execute([StepEntry(s, ids[s][at[s]:at[s] + n]) for s, n in step])
            for (s, n), row in zip(step, logits):
                at[s] += n
                ref = want[s][at[s] - 1]
                assert (row - ref).norm() <= 0.02 * ref.norm(), (s, at[s])
    finally:
        E.GATHER_ROWS = limit


# (lengths, splits, least chunk): tiles of 16 keys and their neighbours, shares that are empty, cluster merge and workspace merge
@pytest.mark.parametrize("Hq,Hkv,D,bs", [(8, 2, 64, 16), (3, 3, 128, 16), (16, 2, 128, 32), (6, 2, 64, 24)])
@pytest.mark.parametrize("lens,splits,chunk", [([1, 15, 16, 17], 1, 16), ([1, 130, 127, 33], 3, 16), ([700, 1, 64, 1030], 8, 16),
                                               ([700, 2000, 5, 65], 12, 16), ([512, 513, 100, 1], 2, 512)])
def test_decode_attention_matches_fp64(Hq, Hkv, D, bs, lens, splits, chunk):
    """Rounding of the result to bf16 (2^-9, doubled) and fp32 weights and sums (2^-20 of values up to about five)."""
    import ctypes
    from trainscale_b200.ops import _lib
    torch.manual_seed(2)
    dev, n, kw = "cuda", len(lens), Hkv * D
    blocks = [-(-k // bs) for k in lens]
    kc, vc = (torch.randn(sum(blocks) + 1, bs, Hkv, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    kc[-1] = vc[-1] = float("nan")              # neither foreign blocks nor the rest of the last one may count
    table = torch.full((n, max(blocks) + 1), sum(blocks), dtype=torch.int32)
    for i, part in enumerate(torch.randperm(sum(blocks)).split(blocks)):
        table[i, :blocks[i]] = part
        if lens[i] % bs:
            kc[part[-1], lens[i] % bs:] = vc[part[-1], lens[i] % bs:] = float("nan")
    table = table.to(dev)
    q = torch.randn(n, Hq * D + 2 * kw, device=dev, dtype=torch.bfloat16)
    out = torch.empty(n, Hq * D, device=dev, dtype=torch.bfloat16)
    po = torch.empty(n, Hq, splits, D, device=dev) if splits > 8 else None
    pl = torch.empty(n, Hq, splits, device=dev) if splits > 8 else None
    lib = _lib.load("decode")
    rc = lib.ts_decode_attention(_lib.ptr(q), q.stride(0), _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), table.shape[1],
                                 _lib.ptr(torch.tensor(lens, dtype=torch.int32, device=dev)), _lib.ptr(out), Hq * D,
                                 _lib.ptr(po), _lib.ptr(pl), n, Hq, Hkv, D, bs, chunk, splits,
                                 ctypes.c_float(1 / math.sqrt(D)), _lib.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    for i, m in enumerate(lens):
        k, v = (c[table[i, :blocks[i]].long()].reshape(-1, Hkv, D)[:m].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,khd->hk", q[i, :Hq * D].double().view(Hq, D), k) / math.sqrt(D), -1)
        ref = torch.einsum("hk,khd->hd", w, v).reshape(-1)
        err = (out[i].double() - ref).abs()
        assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -20 * 5).all(), (i, float(err.max()))


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 2), (128, 3, 1), (16, 20, 20)])
@pytest.mark.parametrize("rows", [1, 37])
def test_rotation_and_cache_write_in_one_launch(D, Hq, Hkv, rows):
    """Against the separate rotation and a scatter; both round a * cos -+ b * sin to bf16 once (2^-8 of the operands)."""
    import ctypes
    from trainscale_b200.ops import _lib, rope
    torch.manual_seed(0)
    cos, sin = rope.rope_tables(512, D, device="cuda")
    qkv = torch.randn(rows, (Hq + 2 * Hkv) * D, device="cuda").bfloat16()
    pos = torch.randint(0, 512, (rows,), device="cuda", dtype=torch.int32)
    slots = torch.randperm(64, device="cuda")[:rows].clone()
    slots[-1] = -1 if rows > 1 else slots[-1]
    want = rope.apply_rope_qkv(qkv.unsqueeze(0), Hq + Hkv, D, cos, sin, pos.unsqueeze(0), rows)[0]
    kc, vc = (torch.full((64, Hkv * D), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    got = qkv.clone()
    rc = _lib.load("decode").ts_rope_cache(_lib.ptr(got), ctypes.c_longlong(got.stride(0)), _lib.ptr(cos), _lib.ptr(sin), _lib.ptr(pos),
                                           _lib.ptr(slots), _lib.ptr(kc), _lib.ptr(vc), ctypes.c_longlong(rows), Hq, Hkv, D,
                                           _lib.stream_ptr())
    assert rc == 0
    assert (got.float() - want.float()).abs().max() <= 2.0 ** -7 * 5
    keep = slots >= 0
    assert torch.equal(kc[slots[keep]], got[keep, Hq * D:(Hq + Hkv) * D]) and torch.equal(vc[slots[keep]], got[keep, (Hq + Hkv) * D:])
    rest = torch.ones(64, dtype=torch.bool, device="cuda")
    rest[slots[keep]] = False
    assert (kc[rest] == 7.0).all() and (vc[rest] == 7.0).all()


@pytest.mark.parametrize("H", [8, 264, 2048, 8192])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_of_step_rows(H, residual):
    """fp32 math on bf16 rows: one rounding of the result, beside a sum in another order (2^-8 covers both)."""
    from trainscale_b200.ops import norm
    torch.manual_seed(0)
    for rows in (1, 5, norm.STEP_ROWS, norm.STEP_ROWS + 1):
        x, r = (torch.randn(rows, H, device="cuda").bfloat16() for _ in range(2))
        w = torch.randn(H, device="cuda").bfloat16()
        y, h = norm.rmsnorm_step(x, w, 1e-5, r if residual else None, 1.0)
        ref, href = norm.rmsnorm_reference(x.double().float(), w.float(), 1e-5, None, 1.0) if not residual else \
            norm.rmsnorm_reference((x.float() + r.float()).bfloat16().float(), w.float(), 1e-5, None, 1.0)
        assert torch.equal(h.float(), href)
        assert ((y.float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-6).all()


def test_chained_steps_wait_for_their_rows():
    """A chain of norm and products whose weights are fetched ahead gives the bits of the same kernels launched one by one."""
    from trainscale_b200.ops import gemm, norm
    torch.manual_seed(0)
    H, I = 2048, 4096
    w1, w2, nw = torch.randn(2 * I, H, device="cuda").bfloat16() * 0.02, torch.randn(H, I, device="cuda").bfloat16() * 0.02, torch.ones(H, device="cuda").bfloat16()
    x = torch.randn(17, H, device="cuda").bfloat16()

    def run(chained):
        h, res = x, None
        for _ in range(20):
            n, res = norm.rmsnorm_step(h, nw, 1e-5, res)
            if not chained:
                torch.cuda.synchronize()
            h = gemm.step_linear(gemm.step_glu(n, w1, "silu", chained=chained), w2, chained=chained)
        return h

    want = run(False)
    for _ in range(5):
        assert torch.equal(run(True), want)


def test_sequences_cross_the_default_rotary_tables():
    """A model that declares 8192 positions, served to 8300: prompt portions and decoding rows on both sides of the border."""
    from trainscale_b200.inference import engine as E
    from trainscale_b200.inference.batch import StepEntry
    from trainscale_b200.models.llama import LlamaConfig, build_model
    cfg = LlamaConfig(vocab_size=300, hidden_size=128, intermediate_size=256, num_hidden_layers=1, num_attention_heads=2,
                      num_key_value_heads=1, head_dim=64)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=1)
    core = E.EngineCore(E.EngineConfig(model="tiny", cache=E.CacheConfig(block_size=16, num_gpu_blocks=600, max_model_len=8300)),
                        model=model)
    assert cfg.max_position_embeddings == 8192 and core.runner.cos.shape[0] >= 8300
    ids = torch.randint(0, 300, (8300,), generator=torch.Generator().manual_seed(3)).tolist()
    want = model(torch.tensor([ids], device="cuda")).logits[0].float().detach()
    at = 0
    for n in (8100, 90, 1, 1, 1, 1, 104, 1, 1):
        row = core.execute([StepEntry(0, ids[at:at + n])])[0]
        at += n
        assert (row - want[at - 1]).norm() <= 0.02 * want[at - 1].norm(), at
    assert at == 8300
    with pytest.raises(ValueError):
        core.execute([StepEntry(0, [1] * (core.runner.cos.shape[0] - at + 1))])


# windows: smaller than a 16-key tile, no multiple of one, of a tile and of a 128-key block; never reached; a cap with and without
@pytest.mark.parametrize("window,softcap", [(5, 0.0), (100, 0.0), (128, 3.0), (500, 0.0), (None, 3.0)])
@pytest.mark.parametrize("graphs", [False, True])
def test_windows_and_capped_scores_on_every_path(window, softcap, graphs):
    """First prompts, portions, decoding rows of their own and beside portions, launched and captured, against the whole-sequence
    forward of the same kernels' training path (bf16 rounding of two layers: 2e-2 of the norm, as above)."""
    from trainscale_b200.inference import engine as E
    from trainscale_b200.inference.batch import StepEntry
    from trainscale_b200.models.llama import LlamaConfig, build_model
    cfg = LlamaConfig(vocab_size=300, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, head_dim=64, sliding_window=window, attn_logit_softcap=softcap, initializer_range=0.1)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=1)
    core = E.EngineCore(E.EngineConfig(model="tiny", enforce_eager=not graphs,
                                       cache=E.CacheConfig(block_size=16, num_gpu_blocks=256, max_model_len=1024)), model=model)
    g = torch.Generator().manual_seed(3)
    ids = {s: torch.randint(0, 300, (n,), generator=g).tolist() for s, n in ((0, 450), (1, 150))}
    want = {s: model(torch.tensor([t], device="cuda")).logits[0].float().detach() for s, t in ids.items()}
    at = {s: 0 for s in ids}
    for step in ([(0, 210), (1, 90)], [(0, 1), (1, 1)], [(0, 130), (1, 1)], [(0, 1), (1, 40)], [(0, 1), (1, 1)], [(0, 99), (1, 7)],
                 [(0, 1), (1, 1)]):
        logits = core.execute([StepEntry(s, ids[s][at[s]:at[s] + n]) for s, n in step])
        for (s, n), row in zip(step, logits):
            at[s] += n
            ref = want[s][at[s] - 1]
            assert (row - ref).norm() <= 0.02 * ref.norm(), (s, at[s])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lens,splits,window,softcap", [([1, 16, 17, 700], 1, 16, 0.0), ([5, 130, 127, 900], 3, 100, 2.0),
                                                        ([2000, 63, 65, 64], 8, 1001, 0.0), ([2000, 1500, 20, 64], 12, 1500, 0.0),
                                                        ([300, 20, 1, 64], 2, 0, 1.5)])
def test_decode_attention_of_a_window_matches_fp64(D, lens, splits, window, softcap):
    """Bounds as without a window; keys before it hold NaN in rows that share no tile with visible ones."""
    import ctypes
    from trainscale_b200.ops import _lib
    torch.manual_seed(2)
    dev, bs, Hq, Hkv, n = "cuda", 16, 6, 2, len(lens)
    kw = Hkv * D
    blocks = [-(-k // bs) for k in lens]
    kc, vc = (torch.randn(sum(blocks) + 1, bs, Hkv, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    table = torch.full((n, max(blocks)), sum(blocks), dtype=torch.int32)
    for i, part in enumerate(torch.randperm(sum(blocks)).split(blocks)):
        table[i, :blocks[i]] = part
        first = max(0, lens[i] - window) // bs if window else 0
        kc[part[:first]] = vc[part[:first]] = float("nan")
    table = table.to(dev)
    q = torch.randn(n, Hq * D + 2 * kw, device=dev, dtype=torch.bfloat16)
    out = torch.empty(n, Hq * D, device=dev, dtype=torch.bfloat16)
    po, pl = torch.empty(n, Hq, splits, D, device=dev), torch.empty(n, Hq, splits, device=dev)
    rc = _lib.load("decode").ts_decode_attention_ex(
        _lib.ptr(q), q.stride(0), _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), table.shape[1],
        _lib.ptr(torch.tensor(lens, dtype=torch.int32, device=dev)), _lib.ptr(out), Hq * D, _lib.ptr(po), _lib.ptr(pl), n, Hq, Hkv, D,
        bs, 16, splits, ctypes.c_float(1 / math.sqrt(D)), window, ctypes.c_float(softcap), _lib.stream_ptr())
    assert rc == 0
    for i, m in enumerate(lens):
        lo = max(0, m - window) if window else 0
        k, v = (c[table[i, :blocks[i]].long()].reshape(-1, Hkv, D)[lo:m].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        sc = torch.einsum("hd,khd->hk", q[i, :Hq * D].double().view(Hq, D), k) / math.sqrt(D)
        if softcap:
            sc = softcap * torch.tanh(sc / softcap)
        ref = torch.einsum("hk,khd->hd", torch.softmax(sc, -1), v).reshape(-1)
        err = (out[i].double() - ref).abs()
        assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -20 * 5).all(), (i, float(err.max()))


# up to four heads per key head share the rows of the matrix instruction with their third parts, more need a second product
@pytest.mark.parametrize("Hq,Hkv", [(4, 1), (8, 1), (6, 2), (10, 2)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("splits", [1, 2, 12])
def test_decode_weights_keep_fp32(Hq, Hkv, D, splits):
    """One key with weight w and value -1 against three with weight 1 whose values add up to w: what is left shows the error of the
    weight.  fp32 leaves 2^-22 of it for the exponential and its argument (sums below two, so 2^-22 for each of two sums), 16 bits
    would leave up to 2^-18."""
    import ctypes
    from trainscale_b200.ops import _lib
    dev, bs, n = "cuda", 16, 24
    kc, vc = (torch.zeros(n * 3, bs, Hkv, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    table = torch.arange(n * 3, dtype=torch.int32, device=dev).view(n, 3)
    q = torch.zeros(n, Hq, D, device=dev, dtype=torch.bfloat16)
    q[..., 0] = math.sqrt(D) if D == 64 else 1.0
    scale = 1 / math.sqrt(D) if D == 64 else 1.0                    # scores are the keys' first values
    s = -(0.1 + 0.6 * torch.rand(n, Hkv, generator=torch.Generator().manual_seed(5))).bfloat16().to(dev)
    at = (3, 7, 8, 14)                  # three keys of weight 1, the one of weight w: in one tile, whose weights share a maximum
    kc[:, :, :, 0] = -100.0                                         # the others do not count
    rows_k, rows_v = kc.view(n, 3 * bs, Hkv, D), vc.view(n, 3 * bs, Hkv, D)
    left = torch.exp(s.double())
    for j in at[:3]:
        rows_k[:, j, :, 0] = 0.0
        part = left.bfloat16()
        rows_v[:, j] = part.unsqueeze(-1)
        left = left - part.double()
    rows_k[:, at[3], :, 0] = s
    rows_v[:, at[3]] = -1.0
    out = torch.empty(n, Hq * D, device=dev, dtype=torch.bfloat16)
    po, pl = torch.empty(n, Hq, splits, D, device=dev), torch.empty(n, Hq, splits, device=dev)
    rc = _lib.load("decode").ts_decode_attention(
        _lib.ptr(q), Hq * D, _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), 3, _lib.ptr(torch.full((n,), 35, dtype=torch.int32, device=dev)),
        _lib.ptr(out), Hq * D, _lib.ptr(po), _lib.ptr(pl), n, Hq, Hkv, D, bs, 16, splits, ctypes.c_float(scale), _lib.stream_ptr())
    assert rc == 0
    exact = -left / (3 + torch.exp(s.double()))                     # (the values' own rest)
    err = (out.view(n, Hkv, Hq // Hkv, D).double() - exact.view(n, Hkv, 1, 1)).abs()
    assert float(err.max()) <= 3 * 2.0 ** -22 / 3, float(err.max())


@pytest.mark.parametrize("Hq,Hkv,D", [(4, 1, 64), (16, 2, 128), (3, 3, 64)])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("splits", [1, 3, 12])
def test_decode_attention_keeps_infinite_values(Hq, Hkv, D, window, splits):
    """An infinite value that is seen, with a weight that any number of bits may hold, makes its dimension infinite and no other;
    one that is not seen (before the window, in the same tile) none.  The largest weight is one, whose lower parts are zero."""
    import ctypes
    from trainscale_b200.ops import _lib
    torch.manual_seed(4)
    dev, bs, lens = "cuda", 16, [1, 16, 17, 47, 300]
    n, blocks = len(lens), [-(-k // bs) for k in lens]
    kc, vc = (torch.randn(sum(blocks), bs, Hkv, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    table = torch.zeros(n, max(blocks), dtype=torch.int32)
    for i, part in enumerate(torch.randperm(sum(blocks)).split(blocks)):
        table[i, :blocks[i]] = part
    table = table.to(dev)

    def put(i, key, d, value):
        vc[table[i, key // bs], key % bs, :, d] = value

    for i, m in enumerate(lens):
        put(i, m - 1, 3, math.inf)                                        # the last key
        put(i, max(0, m - 20), 5, -math.inf)
        put(i, max(0, m - 12), 6, math.nan)
        if window and m > window and (m - window) % bs:
            put(i, m - window - 1, 7, math.inf)
    q = torch.randn(n, Hq * D, device=dev, dtype=torch.bfloat16)
    out = torch.empty_like(q)
    po, pl = torch.empty(n, Hq, splits, D, device=dev), torch.empty(n, Hq, splits, device=dev)
    rc = _lib.load("decode").ts_decode_attention_ex(
        _lib.ptr(q), Hq * D, _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), table.shape[1],
        _lib.ptr(torch.tensor(lens, dtype=torch.int32, device=dev)), _lib.ptr(out), Hq * D, _lib.ptr(po), _lib.ptr(pl), n, Hq, Hkv, D,
        bs, 16, splits, ctypes.c_float(1 / math.sqrt(D)), window, ctypes.c_float(0), _lib.stream_ptr())
    assert rc == 0
    for i, m in enumerate(lens):
        lo = max(0, m - window) if window else 0
        k, v = (c[table[i, :blocks[i]].long()].reshape(-1, Hkv, D)[lo:m].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,khd->hk", q[i].double().view(Hq, D), k) / math.sqrt(D), -1)
        ref = (w.t().unsqueeze(-1) * v).sum(0).reshape(-1)
        got = out[i].double()
        assert torch.equal(got.isinf() * got.sign(), ref.isinf() * ref.sign()) and torch.equal(got.isnan(), ref.isnan()), (i, m)
        fine = ref.isfinite()
        assert ((got - ref).abs()[fine] <= 2.0 ** -8 * ref.abs()[fine] + 2.0 ** -20 * 5).all(), (i, m)


def _decode(q, q_stride, kc, vc, table, lens, out, Hq, Hkv, D, bs, splits):
    import ctypes
    from trainscale_b200.ops import _lib
    n = len(lens)
    po, pl = torch.empty(n, Hq, splits, D, device="cuda"), torch.empty(n, Hq, splits, device="cuda")
    return _lib.load("decode").ts_decode_attention(
        _lib.ptr(q), q_stride, _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), table.shape[1], _lib.ptr(lens), _lib.ptr(out), Hq * D,
        _lib.ptr(po), _lib.ptr(pl), n, Hq, Hkv, D, bs, 16, splits, ctypes.c_float(1 / math.sqrt(D)), _lib.stream_ptr())


@pytest.mark.parametrize("first,more", [(1, 0), (0, 1), (3, 5), (4, 4)])
@pytest.mark.parametrize("D", [64, 128])
def test_decode_attention_of_unaligned_query_rows(first, more, D):
    """Rows that are no 16-byte vectors give the bits of aligned ones."""
    torch.manual_seed(0)
    Hq, Hkv, bs, n = 4, 2, 16, 3
    kc, vc = (torch.randn(8, bs, Hkv, D, device="cuda").bfloat16() for _ in range(2))
    table = torch.arange(6, dtype=torch.int32, device="cuda").view(3, 2)
    lens = torch.tensor([5, 32, 17], dtype=torch.int32, device="cuda")
    q = torch.randn(n, Hq * D, device="cuda").bfloat16()
    want, got = torch.empty_like(q), torch.empty_like(q)
    assert _decode(q, Hq * D, kc, vc, table, lens, want, Hq, Hkv, D, bs, 1) == 0
    wide = torch.zeros(first + n * (Hq * D + more), device="cuda").bfloat16()
    rows = wide[first:].view(n, Hq * D + more)[:, :Hq * D]
    rows.copy_(q)
    assert _decode(rows, Hq * D + more, kc, vc, table, lens, got, Hq, Hkv, D, bs, 1) == 0
    assert torch.equal(got, want)


@pytest.mark.parametrize("splits", [1, 9])
def test_decode_attention_of_more_sequences_than_a_grid_has(splits):
    torch.manual_seed(0)
    n, Hq, D = 65537, 1, 64
    kc, vc = (torch.randn(3, 16, 1, D, device="cuda").bfloat16() for _ in range(2))
    table = (torch.arange(n, device="cuda") % 3).to(torch.int32).view(n, 1)
    lens = torch.ones(n, dtype=torch.int32, device="cuda")
    q, out = torch.randn(n, D, device="cuda").bfloat16(), torch.empty(n, D, device="cuda", dtype=torch.bfloat16)
    assert _decode(q, D, kc, vc, table, lens, out, Hq, 1, D, 16, splits) == 0
    assert torch.equal(out, vc[table[:, 0].long(), 0, 0])             # one key each


@pytest.mark.parametrize("design,shape", [("lovurax", dict(kv=1)), ("mezilix", dict(experts=4, top=2))])
def test_the_serving_benchmarks_closest_table_covers_the_step(design, shape):
    """Every function that the table of the closest model times is called by a prompt's step and by a decoding one."""
    from trainscale_b200.inference import bench_serving as S
    from trainscale_b200.inference.batch import HostBatch, StepEntry
    z = dict(width=256, layers=2, heads=4, dim=64, ff=384, **shape)
    core = S.make_core(S.DESIGNS[design].closest(z), 4096, 4)
    for entries, lengths in (([StepEntry(0, list(range(300)))], [(0, 300)]), ([StepEntry(0, [1])], [(300, 1)])):
        batch = HostBatch(core.cache, entries).to_device("cuda")
        with S.OpTimer(S.closest_table(z, sum(n for _, n in lengths), lengths, core.runner)) as t, torch.no_grad():
            core.runner.logits(core.runner.forward(batch))
        assert t.missing == []
        ops = t.summary({"hbm_gbs": 6460.0, "bf16_tflops": 1695.0})
        assert {"rms norm", "rotary, cache write", "attention"} <= set(ops) and ops["rms norm"]["calls"] == 2 * 2 + 1


@pytest.mark.parametrize("D,keys", [(64, 40), (128, 700)])
def test_rotation_and_decode_attention_wait_in_a_chain(D, keys):
    """Projection, rotation with cache write, attention and output product launched as a chain, against the same kernels one by one:
    each reads what the one before it wrote, the attention also the row that the rotation has just put into the cache."""
    import ctypes
    from trainscale_b200.ops import _lib, gemm, rope
    torch.manual_seed(0)
    Hq, Hkv, n, bs, H = 8, 2, 17, 16, 2048
    lib, kw, blocks = _lib.load("decode"), Hkv * D, -(-keys // bs)
    wqkv, wo = _scaled((Hq + 2 * Hkv) * D, H), _scaled(H, Hq * D)
    cos, sin = rope.rope_tables(keys, D, device="cuda")
    table = torch.arange(n * blocks, dtype=torch.int32, device="cuda").view(n, blocks)
    lens = torch.full((n,), keys, dtype=torch.int32, device="cuda")
    kc0, vc0 = (torch.randn(n * blocks, bs, Hkv, D, device="cuda").bfloat16() for _ in range(2))
    x0 = torch.randn(n, H, device="cuda").bfloat16()
    splits = lib.ts_decode_splits(n, Hkv, keys)
    assert splits <= 8
    steps = [(torch.full((n,), p, dtype=torch.int32, device="cuda"),
              table[:, p // bs].long() * bs + p % bs) for p in range(keys - 12, keys)]
    torch.cuda.synchronize()

    def run(chained):
        def turn():
            if not chained:
                torch.cuda.synchronize()

        x, kc, vc = x0, kc0.clone(), vc0.clone()
        for pos, slots in steps:
            qkv = gemm.step_linear(x, wqkv, chained=chained)
            turn()
            assert lib.ts_rope_cache(_lib.ptr(qkv), ctypes.c_longlong(qkv.stride(0)), _lib.ptr(cos), _lib.ptr(sin), _lib.ptr(pos),
                                     _lib.ptr(slots), _lib.ptr(kc), _lib.ptr(vc), ctypes.c_longlong(n), Hq, Hkv, D,
                                     _lib.stream_ptr()) == 0
            turn()
            out = torch.empty(n, Hq * D, dtype=torch.bfloat16, device="cuda")
            assert lib.ts_decode_attention(_lib.ptr(qkv), qkv.stride(0), _lib.ptr(kc), _lib.ptr(vc), _lib.ptr(table), blocks,
                                           _lib.ptr(lens), _lib.ptr(out), Hq * D, _lib.ptr(None), _lib.ptr(None), n, Hq, Hkv, D, bs, 16,
                                           splits, ctypes.c_float(1 / math.sqrt(D)), _lib.stream_ptr()) == 0
            turn()
            x = gemm.step_linear(out, wo, chained=chained)
            turn()
        return x, kc, vc

    want = run(False)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(True), want))


def _scaled(rows, cols):
    return (torch.randn(rows, cols, device="cuda") / cols ** 0.5).bfloat16()


@pytest.mark.parametrize("D", [64, 128])
def test_an_infinite_value_stays_in_its_dimension_of_portions(D):
    """Portions of prompts make no number of an infinite value's dimension, and every other one keeps its bits."""
    from trainscale_b200.ops import flash
    torch.manual_seed(0)
    Hq, Hkv, n, m = 4, 2, 40, 200
    kw, i32 = Hkv * D, dict(dtype=torch.int32, device="cuda")
    q = torch.randn(n, Hq * D, device="cuda").bfloat16()
    kv = torch.zeros(256, 2 * kw, device="cuda").bfloat16()
    kv[:m] = torch.randn(m, 2 * kw, device="cuda").bfloat16()

    def run():
        out = torch.empty(n, Hq, D, device="cuda", dtype=torch.bfloat16)
        flash.flash_portions(q, kv[:, :kw], kv[:, kw:], out.view(n, -1), Hq, Hkv, D, torch.tensor([0, n], **i32),
                             torch.tensor([0], **i32), torch.tensor([m], **i32), n, 1 / math.sqrt(D))
        return out

    want = run()
    kv[5, kw + 3] = math.inf                                       # of the first key head
    got = run()
    assert not got[:, :2, 3].isfinite().any()
    got[:, :2, 3] = want[:, :2, 3]
    assert torch.equal(got, want)
