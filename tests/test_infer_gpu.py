"""GPU paged-KV engine: kernels vs their PyTorch references and engine-level agreement between
the bf16 GPU path and the fp32 CPU path on greedy tokens."""
import pytest
import torch

from kharon_b200 import ops
from kharon_b200.infer import InferEngine
from kharon_b200.models import GPT, Config
from kharon_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,H", [(64, 4), (128, 2), (32, 4)])
def test_paged_kernels(hd, H):
    torch.manual_seed(0)
    d, bs, nb, nseq, max_lb = H * hd, 8, 40, 3, 6
    kc = torch.zeros(nb, bs, H, hd, device="cuda", dtype=torch.bfloat16); vc = torch.zeros_like(kc)
    kc2, vc2 = kc.clone(), vc.clone()
    btab = torch.randperm(nb, device="cuda")[:nseq * max_lb].int().view(nseq, max_lb)
    lens = [13, 40, 7]
    # prefill every sequence, then one decode token each
    for phase in range(2):
        tok_pos, tok_slot = [], []
        for s, n in enumerate(lens):
            rng = range(n) if phase == 0 else [n]
            tok_pos += list(rng); tok_slot += [s] * len(rng)
        ntok = len(tok_pos)
        pos = torch.tensor(tok_pos, device="cuda", dtype=torch.int32)
        slot = torch.tensor(tok_slot, device="cuda", dtype=torch.int32)
        qkv = torch.randn(ntok, 3 * d, device="cuda").bfloat16()
        out = torch.empty(ntok, d, device="cuda", dtype=torch.bfloat16); out2 = torch.empty_like(out)
        if phase == 0:
            ops.append_kv(qkv, kc, vc, pos, slot, btab, bs, H, hd, ntok)
        ref.append_kv(qkv, kc2, vc2, pos, slot, btab, bs, H, hd, ntok)
        # decode step: the attention kernel stores the new k, v itself
        ops.paged_attn(qkv, kc, vc, out, pos, slot, btab, bs, H, hd, ntok, 64, append=phase == 1)
        torch.cuda.synchronize()
        assert torch.equal(kc, kc2) and torch.equal(vc, vc2)
        ref.paged_attn(qkv, kc2, vc2, out2, pos, slot, btab, bs, H, hd, ntok)
        err = ((out.float() - out2.float()).norm() / out2.float().norm()).item()
        assert err < 1e-2, err


@pytest.mark.parametrize("hd,H,n_split", [(64, 4, 3), (128, 2, 8)])
def test_split_kv_attention_matches_the_single_range_kernel(hd, H, n_split):
    """Keys cut into ranges with a CTA each and merged by log-sum-exp: same result as one CTA per (token, head),
    for prefill tokens and for a decode step that appends its own k, v; ranges beyond a short context are empty."""
    torch.manual_seed(2)
    d, bs, nb, nseq, max_lb, max_ctx = H * hd, 8, 120, 3, 36, 288
    kc = torch.zeros(nb, bs, H, hd, device="cuda", dtype=torch.bfloat16); vc = torch.zeros_like(kc)
    kc2, vc2 = kc.clone(), vc.clone()
    btab = torch.randperm(nb, device="cuda")[:nseq * max_lb].int().view(nseq, max_lb)
    lens = [201, 40, 5]
    for phase in range(2):
        tok_pos, tok_slot = [], []
        for s_, n in enumerate(lens):
            rng = range(n) if phase == 0 else [n]
            tok_pos += list(rng); tok_slot += [s_] * len(rng)
        ntok = len(tok_pos)
        pos = torch.tensor(tok_pos, device="cuda", dtype=torch.int32)
        slot = torch.tensor(tok_slot, device="cuda", dtype=torch.int32)
        qkv = torch.randn(ntok, 3 * d, device="cuda").bfloat16()
        out = torch.empty(ntok, d, device="cuda", dtype=torch.bfloat16); out2 = torch.empty_like(out)
        scratch = torch.zeros(ntok * H * n_split * (hd + 1), device="cuda")
        if phase == 0:
            ops.append_kv(qkv, kc, vc, pos, slot, btab, bs, H, hd, ntok)
            ops.append_kv(qkv, kc2, vc2, pos, slot, btab, bs, H, hd, ntok)
        ops.paged_attn(qkv, kc, vc, out, pos, slot, btab, bs, H, hd, ntok, max_ctx, append=phase == 1, n_split=n_split,
                       scratch=scratch)
        ops.paged_attn(qkv, kc2, vc2, out2, pos, slot, btab, bs, H, hd, ntok, max_ctx, append=phase == 1)
        torch.cuda.synchronize()
        assert torch.equal(kc, kc2) and torch.equal(vc, vc2)
        err = ((out.float() - out2.float()).norm() / out2.float().norm()).item()
        assert err < 5e-3, (phase, err)
    assert ops.error_word() == 0


def test_split_kv_engine_generates_the_same_tokens():
    cfg = Config(2, 128, 2, 300, 96, 1)
    gpu = GPT(cfg, "cuda", torch.bfloat16); gpu.init_weights(1234); gpu.params.w.mul_(6.0); gpu.sync_bf16()
    prompts = [[5, 17, 3, 9], [9, 1, 44, 23, 8, 61, 2], [70, 1]]
    a, _, _ = InferEngine(gpu, block_size=8, max_seqs=5).generate(prompts, 12)
    e = InferEngine(gpu, block_size=8, max_seqs=5, attn_splits=4)
    assert e.attn_splits == 4
    b, _, _ = e.generate(prompts, 12)
    agree = sum(x == y for s_, t in zip(a, b) for x, y in zip(s_, t)) / sum(len(s_) for s_ in a)
    assert agree > 0.9, agree
    assert ops.error_word() == 0


def test_tensor_core_prefill_of_fresh_prompts_matches_the_paged_kernel():
    """Whole fresh prompts take the training attention kernel (one launch per prompt, ragged lengths); the logits of
    the prefill step and the generated tokens match the paged kernel's."""
    cfg = Config(2, 256, 4, 400, 320, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights(99); m.params.w.mul_(5.0); m.sync_bf16()
    gen = torch.Generator().manual_seed(11)
    prompts = [torch.randint(0, 400, (n,), generator=gen).tolist() for n in (64, 131, 200)]
    out = {}
    for flag in (False, True):
        e = InferEngine(m, block_size=8, max_seqs=4, max_tokens=512, flash_prefill=flag)
        toks, _, _ = e.generate(prompts, 1)            # the prefill step alone
        torch.cuda.synchronize()
        assert (e._fresh is not None) == flag
        out[flag] = (toks, e.logits[:3, :400].float().clone())
        more, _, _ = e.generate(prompts, 10)
        out[flag] += (more,)
    err = ((out[True][1] - out[False][1]).norm() / out[False][1].norm()).item()
    assert err < 2e-2, err
    agree = sum(x == y for s_, t in zip(out[True][2], out[False][2]) for x, y in zip(s_, t)) / sum(len(s_) for s_ in out[True][2])
    assert agree > 0.9, agree
    assert ops.error_word() == 0


def test_sampled_generation_from_captured_steps_matches_eager_launches():
    """Temperature sampling replayed from CUDA graphs (step number and seed read from device memory) draws the
    same tokens as eager launches, and a second generation with another seed differs."""
    cfg = Config(2, 512, 8, 300, 96, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights(5); m.sync_bf16()
    prompts = [[5, 17, 3, 9], [9, 1, 44, 23, 8, 61, 2], [70, 1], [3, 3, 3]]
    outs = {}
    for graphs in (False, True):
        e = InferEngine(m, block_size=8, max_seqs=6, use_graphs=graphs)
        e.set_sampling(1.0, 1234)
        a, _, _ = e.generate(prompts, 16)
        e.set_sampling(1.0, 99)
        b, _, _ = e.generate(prompts, 16)
        e.set_sampling(1.0, 1234)
        e.step_no = 0
        c, _, _ = e.generate(prompts, 16)
        outs[graphs] = (a, b, c)
        assert a != b and a == c
        if graphs:
            assert len(e.graphs) > 0
    assert outs[False][0] == outs[True][0] and outs[False][1] == outs[True][1]
    assert ops.error_word() == 0


def test_sampler_and_gather_and_copy():
    torch.manual_seed(1)
    V, ld, n = 50257, 50304, 5
    lg = torch.randn(n, ld, device="cuda").bfloat16()
    out = torch.zeros(64, device="cuda", dtype=torch.int32)
    ops.sample(lg, V, 0.0, 0, 0, 1, out, n)
    assert torch.equal(out[:n].long(), lg[:, :V].float().argmax(-1))
    # temperature: empirical frequencies of a peaked distribution
    lg2 = torch.full((1, 64), -10.0, device="cuda").bfloat16()
    lg2[0, 3] = 2.0; lg2[0, 9] = 2.0
    hits = torch.zeros(64)
    for step in range(40):
        ops.sample(lg2, 64, 1.0, 5, step, 16, out, 1)
        for t in out[:16].tolist():
            hits[t] += 1
    assert hits[3] > 200 and hits[9] > 200 and hits.sum() - hits[3] - hits[9] < 10
    x = torch.randn(20, 128, device="cuda").bfloat16()
    rows = torch.tensor([3, 19, 0], device="cuda", dtype=torch.int32)
    o = torch.empty(3, 128, device="cuda", dtype=torch.bfloat16)
    ops.gather_rows(x, rows, o, 3)
    assert torch.equal(o, x[rows.long()])
    kc = torch.randn(3, 6, 4, 2, 16, device="cuda").bfloat16(); vc = torch.randn_like(kc)
    k0, v0 = kc.clone(), vc.clone()
    pairs = torch.tensor([1, 4, 2, 5], device="cuda", dtype=torch.int32)
    ops.copy_blocks(kc, vc, pairs, 2)
    assert torch.equal(kc[:, 4], k0[:, 1]) and torch.equal(vc[:, 5], v0[:, 2]) and torch.equal(kc[:, 0], k0[:, 0])


def test_engine_gpu_matches_cpu_greedy_and_graph_replay():
    cfg = Config(2, 128, 2, 300, 96, 1)
    cpu = GPT(cfg, "cpu", torch.float32); cpu.init_weights(1234); cpu.params.w.mul_(6.0)
    gpu = GPT(cfg, "cuda", torch.bfloat16); gpu.init_weights(1234); gpu.params.w.mul_(6.0); gpu.sync_bf16()
    prompts = [[5, 17, 3, 9], [9, 1, 44, 23, 8, 61, 2], [70, 1]]
    e1 = InferEngine(cpu, block_size=8, max_seqs=5)
    e2 = InferEngine(gpu, block_size=8, max_seqs=5)
    a, _, _ = e1.generate(prompts, 10)
    b, st, _ = e2.generate(prompts, 10)
    b2, _, _ = e2.generate(prompts, 10)          # second pass replays the captured graphs
    assert b == b2
    agree = sum(x == y for s, t in zip(a, b) for x, y in zip(s, t)) / sum(len(s) for s in a)
    assert agree > 0.9, agree                      # bf16 may flip a near-tie, never most tokens
    g, st, _ = e2.generate_group(prompts[1], 4, 10)
    assert all(x == g[0] for x in g) and st["prefix_blocks_saved"] == 0 * 3 + 3 * (7 // 8)
    assert ops.error_word() == 0


@pytest.mark.parametrize("d,heads,groups", [(512, 8, (1, 5)), (512, 4, (17,)), (1024, 16, (3, 32)), (2048, 16, (8,))])
def test_persistent_decode_kernel_matches_the_kernel_chain(d, heads, groups):
    """All layers of a decode step in one persistent kernel against the five-kernels-per-layer chain: logits
    of the first decode step after an identical prefill (same rounding points; only the order of fp32
    additions differs), then whole greedy generations, eager and from the captured graph.  Head widths 64
    and 128, one and two 16-row tiles, one to eight warps per work unit."""
    cfg = Config(3, d, heads, 600, 160, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights(77); m.params.w.mul_(4.0); m.sync_bf16()
    assert ops.decode_layers_ok(groups[0], d, heads, d // heads, cfg.seq)
    gen = torch.Generator().manual_seed(3)
    for G in groups:
        prompts = [torch.randint(0, 600, (int(n),), generator=gen).tolist() for n in torch.randint(3, 40, (G,), generator=gen)]
        out = {}
        for name, flag in (("chain", False), ("fused", True)):
            e = InferEngine(m, block_size=8, max_seqs=G + 1, persistent_decode=flag, use_graphs=False)
            e.persistent_max = 32
            assert e.persistent == flag
            toks, _, _ = e.generate(prompts, 2)          # prefill, then one decode step
            torch.cuda.synchronize()
            out[name] = (toks, e.logits[:G, :600].float().clone())
        lc, lf = out["chain"][1], out["fused"][1]
        err = ((lc - lf).norm() / lc.norm()).item()
        assert err < 3e-2, (G, err)
        # the sampled token may differ only where the chain's own top two logits are closer than that error
        picked = lf.argmax(-1)                               # greedy: the token the fused step sampled, row by row
        gap = lc.max(-1).values - lc.gather(1, picked[:, None])[:, 0]
        assert float(gap.max()) <= 3e-2 * float(lc.abs().max()), (G, gap.max().item())
        chain = InferEngine(m, block_size=8, max_seqs=G + 1, persistent_decode=False)
        fused = InferEngine(m, block_size=8, max_seqs=G + 1, persistent_decode=True)
        fused.persistent_max = 32
        a, _, _ = chain.generate(prompts, 24)
        b, _, _ = fused.generate(prompts, 24)
        b2, _, _ = fused.generate(prompts, 24)           # replays the captured step
        assert b == b2
        if G >= 3:                                       # a near-tie may flip one sequence, never most of them
            agree = sum(x == y for s, t in zip(a, b) for x, y in zip(s, t)) / sum(len(s) for s in a)
            assert agree > 0.7, (G, agree)
    assert ops.error_word() == 0


@pytest.mark.parametrize("d,heads,G,ctx", [(256, 8, 1, 9), (256, 4, 32, 40), (512, 16, 2, 300), (768, 12, 6, 70), (1024, 8, 16, 150),
                                           (2048, 16, 31, 33), (4096, 32, 17, 20), (4096, 32, 3, 12)])
def test_persistent_decode_steps_against_the_chain(d, heads, G, ctx):
    """Single decode steps at the kernel's edges: one warp step per slice (d = 256), head widths 32 / 64 / 128, one to four
    row groups, several turns of a phase, contexts of more than four keys per lane group, rows that need two launches
    (d = 2048, 4096).  Same inputs, same rounding points, so the logits differ as two summation orders of bf16 layers do (the
    bound of the test above); the appended keys and values of layer 0 only pass one product and agree to a bf16 step."""
    cfg = Config(2, d, heads, 601, 512, 1)
    m = GPT(cfg, "cuda", torch.bfloat16)
    m.init_weights_device(5)
    m.params.w.mul_(3.0); m.sync_bf16()
    gen = torch.Generator().manual_seed(d + G)
    prompts = [torch.randint(0, 601, (int(n),), generator=gen).tolist() for n in torch.randint(max(1, ctx // 2), ctx + 1, (G,), generator=gen)]
    out = {}
    for flag in (False, True):
        e = InferEngine(m, block_size=5, max_seqs=G + 1, max_tokens=G * ctx + 64, persistent_decode=flag, use_graphs=False)
        e.persistent_max = 32
        assert e.persistent == flag
        e.generate(prompts, 2)                           # prefill, then one decode step
        out[flag] = (e.logits[:G, :601].float().clone(), e.kc[0].float().clone(), e.vc[0].float().clone())
    for i, tol in ((0, 3e-2), (1, 2.0 ** -7), (2, 2.0 ** -7)):
        x, y = out[False][i], out[True][i]
        err = ((x - y).norm() / x.norm()).item()
        assert err < tol, (i, err)
    assert ops.error_word() == 0


@pytest.mark.parametrize("d,heads,G,ctx,seq", [(512, 16, 24, 1500, 2000), (512, 8, 31, 900, 1000), (1024, 8, 30, 40, 100), (256, 8, 3, 2100, 4096),
                                               (512, 16, 12, 70, 4096), (512, 16, 16, 2500, 4096), (256, 8, 32, 700, 4096)])
def test_persistent_decode_attention_over_long_contexts(d, heads, G, ctx, seq):
    """More warps to an attention item than one turn has room for (17 to 32 sequences whose longest context outweighs another turn, and not), and
    four positions a lane group for heads of 32 in models of more than 2048 positions, at short and long contexts.  Bounds of the test above."""
    cfg = Config(2, d, heads, 601, seq, 1)
    m = GPT(cfg, "cuda", torch.bfloat16)
    m.init_weights_device(5)
    m.params.w.mul_(3.0); m.sync_bf16()
    gen = torch.Generator().manual_seed(d + G)
    prompts = [torch.randint(0, 601, (int(n),), generator=gen).tolist() for n in torch.randint(max(1, ctx // 9), ctx + 1, (G,), generator=gen)]
    out = {}
    for flag in (False, True):
        e = InferEngine(m, block_size=16, max_seqs=G + 1, n_blocks=G * (ctx // 16 + 2) + 8, max_tokens=G * ctx + 64, persistent_decode=flag, use_graphs=False)
        e.persistent_max = 32
        e.generate(prompts, 2)                           # prefill, then one decode step
        assert e._fused == flag
        out[flag] = (e.logits[:G, :601].float().clone(), e.kc[0].float().clone(), e.vc[0].float().clone())
    for i, tol in ((0, 3e-2), (1, 2.0 ** -7), (2, 2.0 ** -7)):
        x, y = out[False][i], out[True][i]
        err = ((x - y).norm() / x.norm()).item()
        assert err < tol, (i, err)
    assert ops.error_word() == 0


def test_fp32_engine_on_gpu_is_token_exact():
    """The fp32 configuration on the GPU (fp32 weights, activations and KV pool; products on the
    CUDA-core fp32 kernel) reproduces the fp32 CPU engine token for token -- staggered continuous
    batching, contiguous blocks and a prefix-shared group (reference tests/test_infer.c:67-95)."""
    cfg = Config(2, 128, 4, 256, 64, 1)
    cpu = GPT(cfg, "cpu", torch.float32); cpu.init_weights(1337); cpu.params.w.mul_(4.0)
    gpu = GPT(cfg, "cuda", torch.float32); gpu.init_weights(1337); gpu.params.w.mul_(4.0)
    prompts = [[5, 17, 3, 9, 100, 7], [5, 17, 3, 9, 100, 7, 30, 2, 2, 81], [9, 1, 44, 23, 8, 61, 2, 250, 0, 13], [70, 1, 3]]
    n_new = [20, 16, 24, 28]
    want, _, _ = InferEngine(cpu, block_size=4, max_seqs=16).generate(prompts, n_new, max_active=2)
    for bs, active in ((4, 2), (64, 4), (8, 8)):
        eng = InferEngine(gpu, block_size=bs, max_seqs=16)
        assert eng.kc.dtype == torch.float32
        got, _, _ = eng.generate(prompts, n_new, max_active=active)
        assert got == want, (bs, active)
    g, st, _ = InferEngine(gpu, block_size=4, max_seqs=16).generate_group(prompts[0], 8, 20)
    assert all(x == want[0] for x in g) and st["prefix_blocks_saved"] == 7 * (6 // 4)
    assert ops.error_word() == 0


def test_index_guards_record_a_status_code_instead_of_reading_out_of_range():
    """Token ids / positions outside the embedding tables and positions beyond a sequence's block table are
    caught by the kernels' index guards: status word 8, the offending access clamped or skipped, no fault."""
    V, T, d = 64, 16, 64
    wte = torch.randn(V, d, device="cuda").bfloat16(); wpe = torch.randn(T, d, device="cuda").bfloat16()
    tok = torch.tensor([3, 64, 5, -1], device="cuda", dtype=torch.int32)
    pos = torch.tensor([0, 1, 16, 2], device="cuda", dtype=torch.int32)
    out = torch.zeros(4, d, device="cuda", dtype=torch.bfloat16)
    assert ops.error_word() == 0
    ops.embed_fwd(tok, pos, wte, wpe, out, T)
    torch.cuda.synchronize()
    assert ops.error_word() == 8 and ops.error_word() == 0          # reported once, then cleared
    assert torch.equal(out[0], (wte[3].float() + wpe[0].float()).bfloat16())
    H, hd, bs, max_lb = 2, 64, 4, 2
    kc = torch.zeros(4, bs, H, hd, device="cuda", dtype=torch.bfloat16); vc = torch.zeros_like(kc)
    btab = torch.tensor([[0, 1]], device="cuda", dtype=torch.int32)
    qkv = torch.randn(2, 3 * H * hd, device="cuda").bfloat16()
    p2 = torch.tensor([1, 9], device="cuda", dtype=torch.int32)         # position 9 needs a third block
    sl = torch.zeros(2, device="cuda", dtype=torch.int32)
    ops.append_kv(qkv, kc, vc, p2, sl, btab, bs, H, hd, 2)
    torch.cuda.synchronize()
    assert ops.error_word() == 8
    assert torch.equal(kc[0, 1].reshape(-1), qkv[0, H * hd:2 * H * hd]) and float(kc[2:].abs().max()) == 0.0


@pytest.mark.parametrize("V,ld,off", [(2049, 2056, 0), (50257, 50304, 0), (8193, 8200, 1), (131073, 131080, 0)])
def test_greedy_rows_of_large_vocabularies(V, ld, off):
    """Greedy sampling picks the lowest index of the maximum: ties in every position of a 16-byte piece and across threads,
    NaN ignored, the ragged tail, rows that are not 16-byte aligned, several tokens per row."""
    g = torch.Generator(device="cuda").manual_seed(V)
    buf = torch.randn(6 * ld + 8, device="cuda", generator=g).bfloat16()
    lg = buf[off:off + 6 * ld].view(6, ld)
    for r, (i, j) in enumerate([(0, 1), (5, V - 1), (V - 1, V - 1), (8 * 1024 + 3 if V > 8200 else 77, 8 * 1024 + 9 if V > 8210 else 78), (1023, 1024)]):
        lg[r, j] = 100.0
        lg[r, i] = 100.0
    lg[5, 3] = float("nan")
    out = torch.full((6 * 3,), -1, device="cuda", dtype=torch.int32)
    ops.sample(lg, V, 0.0, 1, 0, 3, out, 6)
    x = lg[:, :V].float().nan_to_num(nan=float("-inf"))
    want = (x == x.max(-1, keepdim=True).values).float().argmax(-1).int().repeat_interleave(3)
    assert torch.equal(out, want)


@pytest.mark.parametrize("hd,H,bs", [(64, 3, 16), (32, 4, 5), (128, 2, 1), (64, 2, 64)])
def test_paged_prefill_tiles(hd, H, bs):
    """Prompt pieces through the tile kernel: runs of 1 to 200 tokens from position 0 and in the middle of a sequence, tile edges,
    one buffer and several, other sequences' blocks full of NaN, tokens beyond the context limit (status 8, rows left alone).
    Against fp64 it must not be further off than the fp32 kernel for single tokens (both round once, to bf16: 2^-9 relative
    at most, 1.7e-3 in the 2-norm)."""
    torch.manual_seed(hd + bs)
    d, cases = H * hd, [(0, 1), (0, 17), (3, 64), (60, 65), (0, 200), (150, 5), (63, 1), (190, 16)]      # (first position, length)
    max_lb = (210 + bs - 1) // bs
    nb = max_lb * (len(cases) + 1)
    kc = torch.full((nb, bs, H, hd), float("nan"), device="cuda").bfloat16(); vc = kc.clone()
    btab = torch.randperm(nb, device="cuda")[:len(cases) * max_lb].int().view(len(cases), max_lb)
    runs, pos, slot = [], [], []
    for s, (p0, n) in enumerate(cases):
        runs.append((len(pos), n))
        pos += list(range(p0, p0 + n)); slot += [s] * n
    ntok = len(pos)
    P, S = torch.tensor(pos, device="cuda", dtype=torch.int32), torch.tensor(slot, device="cuda", dtype=torch.int32)
    qkv = torch.randn(ntok, 3 * d, device="cuda").bfloat16()
    hist = {s: (torch.randn(p0, H, hd, device="cuda").bfloat16(), torch.randn(p0, H, hd, device="cuda").bfloat16()) for s, (p0, n) in enumerate(cases)}
    for s, (p0, n) in enumerate(cases):
        for j in range(p0):
            b = int(btab[s, j // bs])
            kc[b, j % bs], vc[b, j % bs] = hist[s][0][j], hist[s][1][j]
    ops.append_kv(qkv, kc, vc, P, S, btab, bs, H, hd, ntok)
    out, one = torch.full((ntok, d), 7.0, device="cuda").bfloat16(), torch.empty(ntok, d, device="cuda", dtype=torch.bfloat16)
    ops.paged_prefill(qkv, kc, vc, out, P, S, btab, bs, H, hd, runs, 210)
    ops.paged_attn(qkv, kc, vc, one, P, S, btab, bs, H, hd, ntok, 210)
    for s, (p0, n) in enumerate(cases):
        r = runs[s][0]
        x = qkv[r:r + n].double().view(n, 3, H, hd)
        k = torch.cat([hist[s][0].double(), x[:, 1]]); v = torch.cat([hist[s][1].double(), x[:, 2]])
        sc = torch.einsum("nhd,khd->hnk", x[:, 0], k) / hd ** 0.5
        sc = sc.masked_fill(torch.arange(p0 + n, device="cuda")[None, None, :] > (p0 + torch.arange(n, device="cuda"))[None, :, None], float("-inf"))
        want = torch.einsum("hnk,khd->nhd", sc.softmax(-1), v).reshape(n, d)
        e = [((o[r:r + n].double() - want).norm() / want.norm()).item() for o in (out, one)]
        assert e[0] < 2.5e-3 and e[0] <= e[1] * 1.02 + 1e-6, (s, e)
    assert ops.error_word() == 0
    out.fill_(7.0)
    ops.paged_prefill(qkv, kc, vc, out, P, S, btab, bs, H, hd, runs, 100)            # positions 100 and more are refused
    late = P >= 100
    assert ops.error_word(reset=True) == 8
    assert (out[late] == 7.0).all() and not (out[~late] == 7.0).all(-1).any()


@pytest.mark.parametrize("hd,H,bs", [(32, 2, 5), (64, 3, 16), (128, 1, 8)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_paged_prefill_keeps_non_finite_values_behind_the_causal_edge(hd, H, bs, bad):
    """An infinity or NaN in V of a later prompt position (first tile, a tile in the middle, last position) changes no earlier row
    by a bit beyond the order of its sums (bf16 outputs: 2^-8 of the row's largest value), and the rows that see it get what the
    kernel for single tokens gives them: the same infinities and NaNs."""
    torch.manual_seed(hd)
    d, n, max_lb = H * hd, 150, (150 + bs - 1) // bs
    qkv = torch.randn(n, 3 * d, device="cuda").bfloat16()
    pos = torch.arange(n, device="cuda", dtype=torch.int32); slot = torch.zeros_like(pos)
    btab = torch.randperm(max_lb, device="cuda").int().view(1, max_lb)
    def attend(x):
        kc = torch.zeros(max_lb, bs, H, hd, device="cuda").bfloat16(); vc = kc.clone()
        ops.append_kv(x, kc, vc, pos, slot, btab, bs, H, hd, n)
        tile, one = torch.empty(n, d, device="cuda", dtype=torch.bfloat16), torch.empty(n, d, device="cuda", dtype=torch.bfloat16)
        ops.paged_prefill(x, kc, vc, tile, pos, slot, btab, bs, H, hd, [(0, n)], n)
        ops.paged_attn(x, kc, vc, one, pos, slot, btab, bs, H, hd, n, n)
        return tile.float(), one.float()
    clean, _ = attend(qkv)
    for at, col in ((9, 3), (63, 0), (64, hd - 1), (100, 5), (n - 1, 7)):
        x = qkv.clone()
        x[at, 2 * d + col] = bad
        tile, one = attend(x)
        assert ((tile[:at] - clean[:at]).abs().amax(1) <= 2.0 ** -8 * clean[:at].abs().amax(1)).all(), at
        assert torch.equal(tile.isnan(), one.isnan()) and torch.equal(tile.isinf(), one.isinf()), at
        assert not tile[at:, col].isfinite().any()
        fin = one.isfinite()
        assert torch.equal(fin, tile.isfinite()) and ((tile - one)[fin].abs() <= 2.0 ** -7 * one[fin].abs().max()).all()
    assert ops.error_word() == 0


@pytest.mark.parametrize("G", [1, 20])
def test_persistent_decode_does_not_hide_scores_that_overflow(G):
    """Scores that are all -inf (q and k of one head so large that their product overflows) have no softmax: the persistent kernel
    hands on the NaN that the kernel chain gives, not zeros that look like an answer."""
    cfg = Config(2, 512, 8, 300, 32, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(3)
    b = m.params.p["l0.qkv_b"]
    b[:64] = 3e38
    b[512:576] = -3e38
    m.sync_bf16()
    for flag in (False, True):
        e = InferEngine(m, block_size=4, max_seqs=G + 1, persistent_decode=flag, use_graphs=False)
        e.generate([[5 + g] for g in range(G)], 1)          # one-token prompts: a decode step at position 0
        assert e.persistent == flag and e.logits[:G, :300].isnan().all(), flag
    assert ops.error_word() == 0


@pytest.mark.parametrize("d,heads,most", [(256, 8, 32), (1024, 16, 32), (1280, 20, 16), (2048, 16, 16), (3072, 24, 16), (4096, 32, 8)])
def test_decode_steps_that_need_two_launches_take_the_chain(d, heads, most):
    """The persistent kernel takes the step sizes at which one launch holds all sequences and beats the chain; the steps beyond them
    (the chain, from eight rows on with the tensor-core GEMM at the largest widths) give the same logits."""
    cfg = Config(2, d, heads, 601, 64, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(5); m.params.w.mul_(3.0); m.sync_bf16()
    e = InferEngine(m, block_size=5, max_seqs=34, max_tokens=256, use_graphs=False)
    assert e.persistent and e.persistent_max == most <= ops.decode_layers_rows(d)
    prompts = [[(7 * g + i) % 601 for i in range(1 + g % 7)] for g in range(33)]
    for G in (most, most + 1):
        rows = {}
        for limit in (most, 32):
            e.persistent_max = limit
            e.generate(prompts[:G], 2)
            assert e._fused == (G <= min(limit, 32))
            rows[limit] = e.logits[:G, :601].float().clone()
        assert ((rows[32] - rows[most]).norm() / rows[32].norm()).item() < 3e-2
    assert ops.error_word() == 0


def test_long_contexts_of_many_sequences_take_split_attention():
    cfg = Config(1, 512, 16, 300, 4200, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(5)
    e = InferEngine(m, block_size=64, n_blocks=200, max_seqs=18, max_tokens=4400, use_graphs=False)
    for first, G, fused in ((4090, 17, False), (4090, 16, True), (4090 - 20, 17, True)):
        e.generate([[3] * first] + [[5 + g] for g in range(G - 1)], 8)      # the last steps stand at first + 6
        assert e._fused == fused, (first, G)
    assert ops.error_word() == 0


@pytest.mark.parametrize("V", [2049, 16384, 16385, 50257])
@pytest.mark.parametrize("n", [1, 148, 149, 700])
def test_greedy_rows_on_both_sides_of_the_thread_count_rule(V, n):
    """Few and many rows, up to and beyond one turn of loads: 256 and 1024 threads a row pick the lowest index of the maximum.
    Logits of 8 bits tie often."""
    g = torch.Generator(device="cuda").manual_seed(V + n)
    lg = torch.randint(-60, 60, (n, (V + 7) // 8 * 8), device="cuda", generator=g).bfloat16()
    lg[:, V:] = 100.0
    lg[0, V - 1] = 99.0
    out = torch.full((n,), -1, device="cuda", dtype=torch.int32)
    ops.sample(lg, V, 0.0, 1, 0, 1, out, n)
    x = lg[:, :V].float()
    want = torch.where(x == x.max(-1, keepdim=True).values, torch.arange(V, device="cuda"), V).min(-1).values.int()
    assert torch.equal(out, want)


@pytest.mark.parametrize("hd,ntok", [(16, 74), (16, 75), (32, 75), (32, 296), (32, 295), (64, 75)])
@pytest.mark.parametrize("append", [False, True])
def test_paged_attention_warps_per_item(hd, ntok, append):
    """Eight heads at the token counts where four warps an item become two (narrow heads) and two become one: contexts of 1 to 300
    positions side by side in a CTA, one token with a bad position (status 8, its row left alone).  fp32 sums, bf16 outputs."""
    torch.manual_seed(ntok + hd)
    H, bs, max_lb = 8, 16, 20
    d, nb = H * hd, ntok * max_lb
    kc = torch.randn(nb, bs, H, hd, device="cuda").bfloat16(); vc = torch.randn_like(kc)
    btab = torch.randperm(nb, device="cuda").int().view(ntok, max_lb)
    pos = torch.tensor([(i * 37) % 300 for i in range(ntok)], device="cuda", dtype=torch.int32)
    pos[7] = 999
    slot = torch.arange(ntok, device="cuda", dtype=torch.int32)
    qkv = torch.randn(ntok, 3 * d, device="cuda").bfloat16()
    out = torch.full((ntok, d), 7.0, device="cuda").bfloat16()
    k2, v2 = kc.clone(), vc.clone()
    ops.paged_attn(qkv, kc, vc, out, pos, slot, btab, bs, H, hd, ntok, 320, append=append)
    assert ops.error_word(reset=True) == 8 and (out[7] == 7.0).all()
    good = [i for i in range(ntok) if i != 7]
    x = qkv.float().view(ntok, 3, H, hd)
    for i in good:
        n = int(pos[i]) + 1
        b = btab[i].long()
        k, v = k2[b].reshape(-1, H, hd)[:n].float(), v2[b].reshape(-1, H, hd)[:n].float()
        if append:
            k[-1], v[-1] = x[i, 1], x[i, 2]
        p = (torch.einsum("hd,khd->hk", x[i, 0], k) / hd ** 0.5).softmax(-1)
        want = torch.einsum("hk,khd->hd", p, v).reshape(d)
        assert ((out[i].float() - want).norm() / want.norm()).item() < 4e-3, i
    if append:
        i = good[-1]
        b, p = int(btab[i, int(pos[i]) // bs]), int(pos[i]) % bs
        assert torch.equal(kc[b, p], qkv[i, d:2 * d].view(H, hd)) and torch.equal(vc[b, p], qkv[i, 2 * d:].view(H, hd))
    else:
        assert torch.equal(kc, k2) and torch.equal(vc, v2)


@pytest.mark.parametrize("H,hd,decoding,lens,tiles", [(16, 64, 8, [16], False), (16, 64, 8, [47], False), (16, 64, 8, [48], True),
                                                      (16, 128, 8, [60], False), (16, 128, 8, [61], True),
                                                      (16, 64, 1, [9, 40, 24], True), (16, 64, 0, [16], True), (8, 32, 3, [128], False),
                                                      (8, 32, 3, [160], True), (8, 32, 0, [15, 15], False), (4, 128, 0, [128], False),
                                                      (4, 128, 0, [150], True), (4, 16, 0, [200], False)])
def test_prompt_pieces_take_the_tile_kernel_where_it_earns_its_launch(H, hd, decoding, lens, tiles):
    """The row ranges that a step hands to the tile kernel and to the kernel for single tokens cover every row once, and the step's
    attention is the same either way."""
    cfg = Config(1, H * hd, H, 300, 512, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(5)
    e = InferEngine(m, block_size=16, max_seqs=20, max_tokens=1024, use_graphs=False, flash_prefill=False)
    pos = [200 + i for i in range(decoding)] + [p for n in lens for p in range(n)]
    slot = list(range(decoding)) + [decoding + i for i, n in enumerate(lens) for _ in range(n)]
    e.np_meta[e._o_pos:e._o_pos + len(pos)] = pos
    e.np_meta[e._o_slot:e._o_slot + len(slot)] = slot
    got = e._prompt_runs(len(pos), decoding + len(lens))
    assert (got is not None) == tiles
    if tiles:
        runs, rest = got
        rows = sorted([i for r, n in runs for i in range(r, r + n)] + [i for a, b in rest for i in range(a, b)])
        assert rows == list(range(len(pos))) and all(n >= 16 for _, n in runs)


@pytest.mark.parametrize("d,heads", [(256, 8), (512, 8), (768, 6), (1024, 16), (1280, 20)])
def test_persistent_decode_workspace_between_steps_of_other_sizes(d, heads):
    """The activation words of a launch are emptied by the next one: steps of one engine with rising and falling numbers of sequences
    (one to four row tiles, both halves of the workspace, the three line pitches of fc's output) give the logits of the kernel chain (bound
    of the tests above)."""
    cfg = Config(4, d, heads, 601, 64, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(5); m.params.w.mul_(3.0); m.sync_bf16()
    e = InferEngine(m, block_size=5, max_seqs=33, max_tokens=320, use_graphs=False)
    c = InferEngine(m, block_size=5, max_seqs=33, max_tokens=320, persistent_decode=False, use_graphs=False)
    e.persistent_max = 32
    prompts = [[(7 * g + i) % 601 for i in range(2 + g % 7)] for g in range(32)]
    for G in (9, 1, 32, 2, 8, 4, 17, 3):
        got = []
        for eng in (c, e):
            eng.generate(prompts[:G], 2)                     # one decode step: a later one would follow the token chosen here
            got.append(eng.logits[:G, :601].float().clone())
        assert e._fused
        assert ((got[0] - got[1]).norm() / got[0].norm()).item() < 3e-2, G
    assert ops.error_word() == 0


@pytest.mark.parametrize("L,d,heads,V", [(L, 256, h, V) for L, h in ((4, 8), (5, 2), (7, 4)) for V in (257, 1000, 50257)] + [(13, 512, 8, 1000), (9, 1024, 16, 1000)])
def test_persistent_decode_slots_of_many_layers(L, d, heads, V):
    """Models with more layers than an activation has slots.  At width 256 some CTAs of a 148-CTA grid have columns of the head and no part in any layer: without a
    wait they come to the head when the kernel starts, and layers before the last have used the words of its slot.  Logits against the kernel chain, per eight columns (one CTA's share): the norm of
    a block's difference over the mean block's norm.  Two bf16 paths lie 3e-2 apart (the tests above); the worst of 6283 blocks of eight such differences
    is 2.4 times their mean, below 0.2; logits of another layer would be off by about 1."""
    cfg = Config(L, d, heads, V, 64, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(5); m.params.w.mul_(3.0); m.sync_bf16()
    e = InferEngine(m, block_size=5, max_seqs=33, max_tokens=320, use_graphs=False)
    c = InferEngine(m, block_size=5, max_seqs=33, max_tokens=320, persistent_decode=False, use_graphs=False)
    e.persistent_max = 32
    prompts = [[(7 * g + i) % V for i in range(2 + g % 7)] for g in range(32)]
    for G in (1, 8, 32, 1):
        got = []
        for eng in (c, e):
            eng.generate(prompts[:G], 2)                     # one decode step
            got.append(torch.nn.functional.pad(eng.logits[:G, :V].double(), (0, -V % 8)).view(G, -1, 8))
        assert e._fused and not c._fused
        per = (got[0] - got[1]).pow(2).sum((0, 2)).sqrt()
        assert (per / got[0].pow(2).sum((0, 2)).mean().sqrt()).max().item() < 0.2, (G, per.argmax().item())
    assert ops.error_word() == 0


@pytest.mark.parametrize("d,heads,V,G", [(512, 8, 300, 3), (1024, 16, 20000, 9)])
def test_persistent_decode_gives_up_and_recovers(d, heads, V, G):
    """A wait that runs out: the head is asked for a row that is not part of the step, whose words nobody writes.  The launch ends by itself with
    code 9, whether all of its weight copies have been issued by then (few columns) or not, and the launches after it, one for each half of the
    workspace, give the bits of the one before."""
    cfg = Config(5, d, heads, V, 64, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.init_weights_device(5); m.sync_bf16()
    e = InferEngine(m, block_size=5, max_seqs=33, max_tokens=320, use_graphs=False)
    e.persistent_max = 32
    e.generate([[(7 * g + i) % V for i in range(2 + g)] for g in range(G)], 2)
    assert e._fused and ops.error_word() == 0
    want, rows = e.logits[:G, :V].clone(), e.d_rows.clone()
    e.d_rows[G - 1] = G                                      # a row of the workspace, but of no sequence
    e._forward(G, G, 1)
    torch.cuda.synchronize()
    assert ops.error_word() == 9
    e.d_rows.copy_(rows)
    for _ in range(3):
        e.logits.fill_(7.0)
        e._forward(G, G, 1)
        assert torch.equal(e.logits[:G, :V], want)
    assert ops.error_word() == 0


@pytest.mark.parametrize("G", [1, 8, 20])
def test_persistent_decode_hands_zeros_on(G):
    """An empty activation word is zero, so results that are zero travel as {-0.0, +0.0}: a model whose every product is zero neither
    stalls nor differs from the kernel chain."""
    cfg = Config(2, 512, 8, 300, 32, 1)
    m = GPT(cfg, "cuda", torch.bfloat16); m.params.w.zero_(); m.sync_bf16()
    for flag in (False, True):
        e = InferEngine(m, block_size=4, max_seqs=G + 1, persistent_decode=flag, use_graphs=False)
        e.persistent_max = 32
        e.logits.fill_(7.0)
        outs, _, _ = e.generate([[5 + g, 9] for g in range(G)], 3)
        assert e._fused == flag and (e.logits[:G, :300] == 0).all() and all(o[2:] == [0, 0, 0] for o in outs)
        assert (e.kc.float() == 0).all() and (e.vc.float() == 0).all()
    assert ops.error_word() == 0
