"""Numerics of each CUDA kernel against the plain-PyTorch fp32 evaluation of the same op."""
import pytest
import torch

from kharon_b200 import ops
from kharon_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def relerr(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K,bn", [(128, 256, 64, 0), (256, 512, 256, 256), (384, 320, 192, 128), (200, 136, 72, 64),
                                      (1024, 1024, 1024, 0), (8, 1024, 512, 0)])
def test_gemm_majors(a_mn, b_mn, M, N, K, bn):
    torch.manual_seed(0)
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("pitch not 16-byte aligned for this major")
    a = _rand(K, M) if a_mn else _rand(M, K)
    b = _rand(K, N) if b_mn else _rand(N, K)
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, block_n=bn)
    want = torch.empty(M, N, device=DEV)
    ref.gemm(a, b, want, a_mn, b_mn, False, 0, None, None, 1.0)
    torch.cuda.synchronize()
    assert ops.error_word() == 0
    assert relerr(out, want) < 6e-3, relerr(out, want)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 320), (384, 328, 192), (1000, 1024, 1024), (4096, 2048, 512)])
def test_gemm_cta_pairs(a_mn, b_mn, M, N, K):
    """256 x 256 tiles on CTA pairs (cta_group::2) against the PyTorch product, ragged edges included."""
    torch.manual_seed(10)
    a = _rand(K, M) if a_mn else _rand(M, K)
    b = _rand(K, N) if b_mn else _rand(N, K)
    bias, resid = _rand(N), _rand(M, N)
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, block_n=512, epi=ops.EPI_BIAS_RESID, bias=bias, aux=resid)
    want = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ref.gemm(a, b, want, a_mn, b_mn, False, ops.EPI_BIAS_RESID, bias, resid, 1.0)
    torch.cuda.synchronize()
    assert ops.error_word() == 0
    assert relerr(out, want) < 6e-3, relerr(out, want)
    acc = torch.ones(M, N, device=DEV)
    ops.gemm(a, b, acc, a_mn=a_mn, b_mn=b_mn, block_n=512, accumulate=True)
    wf = torch.empty(M, N, device=DEV)
    ref.gemm(a, b, wf, a_mn, b_mn, False, 0, None, None, 1.0)
    assert relerr(acc, 1 + wf) < 1e-4


def test_gemm_fp32_accumulate_and_alpha():
    torch.manual_seed(1)
    M, N, K = 256, 384, 320
    a, b = _rand(K, M), _rand(K, N)
    out = torch.randn(M, N, device=DEV)
    base = out.clone()
    ops.gemm(a, b, out, a_mn=True, b_mn=True, accumulate=True, alpha=0.5)
    want = base + 0.5 * (a.float().t() @ b.float())
    assert relerr(out, want) < 1e-5
    ops.gemm(a, b, out, a_mn=True, b_mn=True, accumulate=False)
    assert relerr(out, a.float().t() @ b.float()) < 1e-5


@pytest.mark.parametrize("M,N,K,bn", [(256, 256, 64, 0), (384, 328, 200, 256), (2048, 512, 4096, 512), (1000, 1024, 1032, 0),
                                      (136, 64, 72, 64), (3072, 2048, 2048, 0), (512, 1536, 640, 128)])
def test_gemm_weight_gradient_with_bias_gradient(M, N, K, bn):
    """dW += dY^T X with db += column sums of dY taken from the operand tiles in shared memory
    (single tiles, CTA pairs, ragged M / N / K, several tiles per CTA) against PyTorch."""
    torch.manual_seed(12)
    dy, x = _rand(K, M), _rand(K, N)
    dw = torch.randn(M, N, device=DEV)
    db = torch.randn(M, device=DEV)
    want_w = dw + dy.float().t() @ x.float()
    want_b = db + dy.float().sum(0)
    ops.gemm(dy, x, dw, a_mn=True, b_mn=True, accumulate=True, block_n=bn, colsum=db)
    torch.cuda.synchronize()
    assert ops.error_word() == 0
    assert relerr(dw, want_w) < 1e-4, relerr(dw, want_w)
    assert relerr(db, want_b) < 1e-5, relerr(db, want_b)
    # overwrite form, and run-to-run identical bits
    db2, db3 = torch.full((M,), 3.0, device=DEV), torch.full((M,), -1.0, device=DEV)
    ops.gemm(dy, x, dw, a_mn=True, b_mn=True, block_n=bn, colsum=db2)
    ops.gemm(dy, x, dw, a_mn=True, b_mn=True, block_n=bn, colsum=db3)
    assert torch.equal(db2, db3) and relerr(db2, dy.float().sum(0)) < 1e-5


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("split", [2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(128, 64, 512), (200, 72, 1000), (8, 136, 4104), (513, 257, 1496), (256, 512, 9216)])
def test_gemm_split_over_a_cluster(M, N, K, split, bn):
    """K split over the CTAs of a cluster: whole and ragged tiles, K remainders, slices of unequal length, with every
    epilogue.  fp32 sums of K products in another order differ by at most K * 2^-24 of the sum of magnitudes, which for
    normal operands is about sqrt(K) times the result: 1e-5 and 2e-4 leave a factor of ten; bf16 outputs round at 2^-9."""
    torch.manual_seed(M + N + K)
    pad = lambda n: (n + 7) // 8 * 8
    r = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    blk = 4096 * split + bn
    dy, x = r(K, pad(M))[:, :M], r(K, pad(N))[:, :N]
    want = dy.double().t() @ x.double()
    dw = torch.ones(M, pad(N), device="cuda")[:, :N]
    db = torch.ones(M, device="cuda")
    ops.gemm(dy, x, dw, a_mn=True, b_mn=True, accumulate=True, colsum=db, block_n=blk)
    assert ((dw - 1 - want).norm() / want.norm()).item() < 1e-5
    cs = dy.double().sum(0)
    assert ((db - 1 - cs).norm() / cs.norm()).item() < 2e-4
    again = torch.ones(M, pad(N), device="cuda")[:, :N]
    ops.gemm(dy, x, again, a_mn=True, b_mn=True, accumulate=True, block_n=blk)
    assert torch.equal(again, dw)
    a, w = r(M, pad(K))[:, :K], r(N, pad(K))[:, :K]
    bias, aux = r(pad(N))[:N], r(M, pad(N))[:, :N]
    acc = a.double() @ w.double().t()
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID, ops.EPI_DGELU, ops.EPI_RESID):
        out = torch.full((M, pad(N)), 7.0, device="cuda").bfloat16()
        ax = aux.clone() if epi != ops.EPI_BIAS_GELU else torch.empty(M, pad(N), device="cuda", dtype=torch.bfloat16)[:, :N]
        if epi == ops.EPI_NONE or epi == ops.EPI_BIAS:
            ax = None
        elif epi != ops.EPI_BIAS_GELU:
            ax = torch.zeros(M, pad(N), device="cuda", dtype=torch.bfloat16)[:, :N].copy_(aux)
        ops.gemm(a, w, out[:, :N], epi=epi, bias=bias if epi in (ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID) else None,
                 aux=ax, block_n=blk)
        one = torch.full((M, pad(N)), 7.0, device="cuda").bfloat16()
        ax1 = None if ax is None else torch.zeros(M, pad(N), device="cuda", dtype=torch.bfloat16)[:, :N].copy_(aux)
        ops.gemm(a, w, one[:, :N], epi=epi, bias=bias if epi in (ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID) else None,
                 aux=ax1, block_n=bn)
        err = ((out[:, :N].double() - one[:, :N].double()).norm() / one[:, :N].double().norm()).item()
        assert err < 2.0 ** -8, (epi, err)
        assert torch.equal(out[:, N:], one[:, N:])
        if epi == ops.EPI_NONE:
            assert ((out[:, :N].double() - acc).norm() / acc.norm()).item() < 2.0 ** -8
    assert ops.error_word() == 0


@pytest.mark.parametrize("M,N,K,blk", [(200, 72, 1000, 4096 * 2 + 64), (513, 257, 1496, 4096 * 4 + 128), (130, 136, 4104, 4096 * 8 + 64),
                                       (200, 328, 1032, 256), (520, 264, 2048, 512), (200, 72, 1032, 64)])
def test_gemm_gelu_stores_the_pre_activation(M, N, K, blk):
    """The second output of the GELU epilogue (read by the backward pass) from split, wide and paired tiles, whole and ragged columns:
    the bf16 of acc + bias, nothing outside the M x N block, and the output is the GELU of exactly that bf16 value."""
    torch.manual_seed(M + K)
    pad = (N + 7) // 8 * 8 + 8
    a, w = _rand(M, K, scale=0.3), _rand(N, K, scale=0.1)
    bias = _rand(pad)[:N]
    out, aux = torch.full((M + 3, pad), 7.0, device=DEV).bfloat16(), torch.full((M + 3, pad), 5.0, device=DEV).bfloat16()
    ops.gemm(a, w, out[:M, :N], epi=ops.EPI_BIAS_GELU, bias=bias, aux=aux[:M, :N], block_n=blk)
    pre = (a.double() @ w.double().t() + bias.double())
    assert ((aux[:M, :N].double() - pre).abs() <= 2.0 ** -8 * pre.abs() + 1e-4).all()       # one rounding; fp32 sums of K products
    x = aux[:M, :N].float()
    want = 0.5 * x * (1 + torch.tanh(0.7978845608 * (x + 0.044715 * x ** 3)))
    assert ((out[:M, :N].float() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-3).all()      # and the kernel's approximate tanh
    for t, v in ((out, 7.0), (aux, 5.0)):
        assert (t[M:] == v).all() and (t[:M, N:] == v).all()
    assert ops.error_word() == 0


@pytest.mark.parametrize("M,N,bn", [(7680, 2048, 256), (7700, 2000, 512)])
@pytest.mark.parametrize("K", [1032, 2048])
def test_gemm_long_k_tiles(M, N, K, bn):
    """K beyond 1024 without column sums: four epilogue warps with all columns of a tile (single tiles and CTA pairs), at least three
    tiles a worker so that both accumulator buffers come round, every epilogue of the training step and fp32 accumulation."""
    torch.manual_seed(K)
    a, w, bias = _rand(M, K, scale=0.3), _rand(N, K, scale=0.1), _rand(N)
    aux = _rand(M, N)
    acc = a.float() @ w.float().t()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID, ops.EPI_DGELU, ops.EPI_RESID):
        ax, ax_ref = aux.clone(), aux.clone()
        want = torch.empty_like(out)
        ops.gemm(a, w, out, epi=epi, bias=bias, aux=ax, block_n=bn)
        ref.gemm(a, w, want, False, False, False, epi, bias, ax_ref, 1.0)
        assert relerr(out, want) < 8e-3, epi
        assert relerr(ax, ax_ref) < 8e-3, epi
    base = torch.randn(M, N, device=DEV)
    c = base.clone()
    ops.gemm(a, w, c, accumulate=True, alpha=0.5, block_n=bn)
    assert relerr(c - base, 0.5 * acc) < 1e-4          # fp32 sums of K products and one addition to values of size one
    assert ops.error_word() == 0


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_gemm_f32_oracle_kernel(ta, tb):
    torch.manual_seed(13)
    M, N, K = 150, 77, 203
    A = torch.randn(K, M, device=DEV).t() if ta else torch.randn(M, K, device=DEV)
    B = torch.randn(N, K, device=DEV).t() if tb else torch.randn(K, N, device=DEV)
    got = ops._matmul_f32(A, B)
    want = (A.double() @ B.double()).float()
    assert relerr(got, want) < 2e-6


@pytest.mark.parametrize("epi", [ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID, ops.EPI_DGELU, ops.EPI_RESID])
@pytest.mark.parametrize("N", [512, 328])
def test_gemm_epilogues(epi, N):
    torch.manual_seed(2)
    M, K = 320, 256
    a, b = _rand(M, K, scale=0.5), _rand(N, K, scale=0.1)
    bias = _rand(N)
    aux = _rand(M, N)
    aux_ref = aux.clone()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    want = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, out, epi=epi, bias=bias, aux=aux)
    ref.gemm(a, b, want, False, False, False, epi, bias, aux_ref, 1.0)
    assert relerr(out, want) < 8e-3
    if epi == ops.EPI_BIAS_GELU:
        assert relerr(aux, aux_ref) < 8e-3


def test_gemm_vocab_shapes():
    """Head shapes: N = 50257 (ragged), and the M-major weight-gradient with M = 50304 padded."""
    torch.manual_seed(3)
    R, d, V, Vp = 256, 128, 50257, 50304
    x, wte = _rand(R, d), _rand(V, d, scale=0.05)
    logits = torch.zeros(R, Vp, device=DEV, dtype=torch.bfloat16)
    ops.gemm(x, wte, logits[:, :V])
    want = x.float() @ wte.float().t()
    assert relerr(logits[:, :V], want) < 6e-3
    assert logits[:, V:].abs().max().item() == 0
    dl = _rand(R, Vp, scale=0.01)
    dl[:, V:] = 0
    dx = torch.empty(R, d, device=DEV, dtype=torch.bfloat16)
    ops.gemm(dl[:, :V], wte, dx, b_mn=True)
    assert relerr(dx, dl[:, :V].float() @ wte.float()) < 6e-3
    dw = torch.zeros(V, d, device=DEV)
    ops.gemm(dl[:, :V], x, dw, a_mn=True, b_mn=True, accumulate=True)
    assert relerr(dw, dl[:, :V].float().t() @ x.float()) < 1e-4


def test_layernorm_fwd_bwd():
    torch.manual_seed(4)
    for rows, d in [(64, 128), (1000, 512), (4096, 2048)]:
        x, w, b = _rand(rows, d), _rand(d), _rand(d)
        dy, dres = _rand(rows, d), _rand(rows, d)
        y = torch.empty_like(x); mean = torch.empty(rows, device=DEV); rstd = torch.empty(rows, device=DEV)
        ops.layernorm_fwd(x, w, b, y, mean, rstd)
        y2 = torch.empty_like(x); m2 = torch.empty_like(mean); r2 = torch.empty_like(rstd)
        ref.layernorm_fwd(x, w, b, y2, m2, r2)
        assert relerr(y, y2) < 4e-3 and relerr(mean, m2) < 1e-4 and relerr(rstd, r2) < 1e-4
        dx = torch.empty_like(x); dw = torch.ones(d, device=DEV); db = torch.ones(d, device=DEV)
        part = torch.zeros(ops.layernorm_bwd_scratch_elems(rows, d), device=DEV)
        ops.layernorm_bwd(dy, x, w, mean, rstd, dres, dx, dw, db, part)
        dx2 = torch.empty_like(x); dw2 = torch.ones(d, device=DEV); db2 = torch.ones(d, device=DEV)
        ref.layernorm_bwd(dy, x, w, m2, r2, dres, dx2, dw2, db2)
        assert relerr(dx, dx2) < 5e-3 and relerr(dw, dw2) < 1e-3 and relerr(db, db2) < 1e-3


def test_xent_vocab_slices_combine_to_full_softmax():
    """Per-slice statistics + combined gradient equal the full-row cross-entropy."""
    torch.manual_seed(6)
    R, V, parts = 96, 1003, 2
    vs = (V + parts - 1) // parts
    ld = (vs + 63) // 64 * 64
    full = _rand(R, V, scale=2.0)
    tgt = torch.randint(0, V, (R,), device=DEV, dtype=torch.int32)
    tgt[5] = -1
    stats, bufs = [], []
    for r in range(parts):
        v0, v1 = r * vs, min(V, (r + 1) * vs)
        lg = torch.full((R, ld), 77.0, device=DEV, dtype=torch.bfloat16)
        lg[:, :v1 - v0] = full[:, v0:v1]
        st = torch.empty(R, 3, device=DEV); st2 = torch.empty(R, 3, device=DEV)
        ops.xent_stats(lg, v1 - v0, tgt, v0, st)
        ref.xent_stats(lg, v1 - v0, tgt, v0, st2)
        assert torch.equal(torch.isinf(st[:, 2]), torch.isinf(st2[:, 2]))
        fin = ~torch.isinf(st2[:, 2])
        assert relerr(st[:, :2], st2[:, :2]) < 1e-3 and relerr(st[fin, 2], st2[fin, 2]) < 1e-6
        stats.append(st); bufs.append((lg, v0, v1))
    sa = torch.stack(stats)
    gm = sa[..., 0].max(0).values
    gs = (sa[..., 1] * torch.exp(sa[..., 0] - gm)).sum(0)
    loss = torch.where(tgt >= 0, torch.log(gs) + gm - sa[..., 2].max(0).values, torch.zeros_like(gm))
    want = full.clone().float()
    lp = torch.log_softmax(want, -1)
    want_loss = torch.where(tgt >= 0, -lp.gather(1, tgt.clamp(min=0).long()[:, None]).squeeze(1), torch.zeros(R, device=DEV))
    assert relerr(loss, want_loss) < 1e-3
    grad = torch.softmax(want, -1)
    grad[torch.arange(R, device=DEV), tgt.clamp(min=0).long()] -= 1.0
    grad[tgt < 0] = 0
    grad *= 0.25
    for lg, v0, v1 in bufs:
        ops.xent_grad(lg, v1 - v0, tgt, v0, gm, gs, uniform=0.25)
        assert relerr(lg[:, :v1 - v0], grad[:, v0:v1]) < 1e-2
        pad8 = (v1 - v0 + 7) // 8 * 8
        assert lg[:, v1 - v0:pad8].abs().max().item() == 0 if pad8 > v1 - v0 else True


def test_xent():
    torch.manual_seed(5)
    for R, V, ld in [(64, 256, 256), (130, 50257, 50304), (32, 1000, 1008)]:
        logits = torch.zeros(R, ld, device=DEV, dtype=torch.bfloat16)
        logits[:, :V] = _rand(R, V, scale=2.0)
        logits[:, V:] = 99.0   # padding must be ignored
        tgt = torch.randint(0, V, (R,), device=DEV, dtype=torch.int32)
        tgt[3] = -1
        coef = torch.randn(R, device=DEV)
        l2 = logits.clone()
        rl = torch.empty(R, device=DEV); pr = torch.empty(R, device=DEV)
        rl2 = torch.empty(R, device=DEV); pr2 = torch.empty(R, device=DEV)
        ops.xent(logits, V, tgt, coef=coef, rowloss=rl, prob=pr)
        ref.xent(l2, V, tgt, coef, 1.0, rl2, pr2, True)
        assert relerr(rl, rl2) < 1e-3 and relerr(pr, pr2) < 2e-3
        assert relerr(logits, l2) < 1e-2
        if ld > V:
            assert logits[:, V:].abs().max().item() == 0
        assert logits[3].abs().max().item() == 0


@pytest.mark.parametrize("R,V,ld", [(1, 1, 8), (9, 7, 8), (17, 250, 256), (8, 256, 256), (33, 257, 264), (7, 512, 520), (40, 1023, 1024), (25, 1030, 1032),
                                    (11, 2041, 2048), (6, 2048, 2056), (7, 9001, 9008), (600, 2500, 2504)])
def test_xent_short_rows(R, V, ld):
    """A warp per row up to 2048 columns, a CTA per row past them (the last three shapes; the last with 256 threads): every number of pieces a lane, odd vocabularies, NaN in the
    padding, masked (-inf) logits, rows without a target; loss, probability and gradient against fp64, the gradient rounded once to bf16."""
    torch.manual_seed(R + V)
    x = torch.full((R, ld), float("nan"), device=DEV).bfloat16()
    x[:, :V] = _rand(R, V, scale=3.0)
    if V > 16:
        x[:, V // 2:V // 2 + 9] = float("-inf")
    t = torch.randint(0, max(V // 2, 1), (R,), device=DEV, dtype=torch.int32)
    if R > 5:
        t[5], t[4] = -1, V
    coef = torch.randn(R, device=DEV)
    rl, pr, g = torch.empty(R, device=DEV), torch.empty(R, device=DEV), x.clone()
    ops.xent(g, V, t, coef=coef, rowloss=rl, prob=pr, write_grad=False)
    assert torch.equal(g.view(torch.int16), x.view(torch.int16))
    rl2, pr2 = torch.empty_like(rl), torch.empty_like(pr)
    ops.xent(g, V, t, coef=coef, rowloss=rl2, prob=pr2)
    assert torch.equal(rl, rl2) and torch.equal(pr, pr2)
    ok = (t >= 0) & (t < V)
    p = x[:, :V].double().softmax(1)
    pt = p.gather(1, t.clamp(0, V - 1).long()[:, None])[:, 0]
    assert relerr(rl, torch.where(ok, -pt.log(), 0.)) < 1e-5 and relerr(pr, torch.where(ok, pt, 0.)) < 1e-5       # fp32 sums of up to 9001 terms
    want = p.clone()
    want[torch.arange(R, device=DEV)[ok], t[ok].long()] -= 1
    want *= torch.where(ok, coef.double(), 0.)[:, None]
    assert ((g[:, :V].double() - want).abs() <= want.abs() * 2 ** -8 + 1e-5 * coef.abs()[:, None]).all()
    assert not g[:, V:].any()


@pytest.mark.parametrize("V", [16390, 9001, 5000, 2000, 1000, 600, 300])
def test_xent_bits_of_a_row_do_not_depend_on_the_call(V):
    """Loss, probability and gradient of a row have the same bits with and without the gradient and beside few or many rows: past 592 to 1776 rows a row
    is summed by 256 threads, without the gradient or up to 16384 columns, else by 512; up to 1024 columns by one warp past 1024 rows, else by two."""
    torch.manual_seed(V)
    ld, rows = (V + 7) // 8 * 8, 1900
    x = torch.zeros(rows, ld, device=DEV).bfloat16()
    x[:, :V] = _rand(rows, V, scale=4.0)
    x[3, :V // 2] = float("-inf")
    t = torch.randint(V // 2, V, (rows,), device=DEV, dtype=torch.int32)
    out = []
    for n, grad in ((rows, True), (rows, False), (40, True), (40, False)):
        g, rl, pr = x[:n].clone(), torch.empty(n, device=DEV), torch.empty(n, device=DEV)
        ops.xent(g, V, t[:n], rowloss=rl, prob=pr, write_grad=grad)
        out.append((rl, pr, g))
    for i, (rl, pr, g) in enumerate(out):
        n = rl.numel()
        assert torch.equal(rl, out[0][0][:n]) and torch.equal(pr, out[0][1][:n])
        assert torch.equal(g, (x if i & 1 else out[0][2])[:n])
    want = -x[:, :V].double().log_softmax(1).gather(1, t.long()[:, None])[:, 0]
    assert relerr(out[0][0], want) < 1e-5


def test_adamw_matches_torch_and_emits_bf16():
    torch.manual_seed(6)
    n = 100003
    p = torch.randn(n + 1, device=DEV)[:n]
    p = torch.randn(n, device=DEV); g = torch.randn(n, device=DEV)
    m = torch.zeros(n, device=DEV); v = torch.zeros(n, device=DEV)
    pb = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    pt = torch.nn.Parameter(p.clone()); pt.grad = g.clone()
    opt = torch.optim.AdamW([pt], lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in (1, 2, 3):
        gg = g.clone()
        ops.adamw(p, gg, m, v, pb, lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, wd=0.1, step=step)
        assert gg.abs().max().item() == 0
        opt.step()
        assert torch.allclose(p, pt.data, rtol=1e-5, atol=1e-6)
        assert torch.equal(pb, p.to(torch.bfloat16))


def test_embed_and_colsum():
    torch.manual_seed(7)
    B, T, d, V = 4, 64, 128, 300
    tok = torch.randint(0, V, (B * T,), device=DEV, dtype=torch.int32)
    tok[5] = tok[17] = tok[200] = 11
    wte, wpe = _rand(V, d), _rand(T, d)
    out = torch.empty(B * T, d, device=DEV, dtype=torch.bfloat16)
    ops.embed_fwd(tok, None, wte, wpe, out, T)
    want = torch.empty_like(out); ref.embed_fwd(tok, None, wte, wpe, want, T)
    assert relerr(out, want) < 4e-3
    dx = _rand(B * T, d)
    dwte = torch.ones(V, d, device=DEV); dwpe = torch.ones(T, d, device=DEV)
    ops.embed_bwd(tok, dx, dwte, dwpe, B, T)
    dwte2 = torch.ones(V, d, device=DEV); dwpe2 = torch.ones(T, d, device=DEV)
    ref.embed_bwd(tok, dx, dwte2, dwpe2, B, T)
    assert relerr(dwte, dwte2) < 1e-5 and relerr(dwpe, dwpe2) < 1e-5
    for rows, N in [(777, 322), (4096, 2048), (100, 64)]:
        x = _rand(rows, (N + 7) // 8 * 8)[:, :N]
        cs = torch.ones(N, device=DEV)
        ops.colsum(x, cs, accumulate=True)
        assert relerr(cs, 1 + x.float().sum(0)) < 1e-5


@pytest.mark.parametrize("B,T,H,hd", [(2, 256, 4, 64), (1, 512, 2, 128), (3, 64, 2, 64), (2, 200, 2, 128), (1, 1024, 1, 64),
                                      (2, 384, 3, 128), (1, 130, 2, 64), (40, 512, 8, 128), (5, 72, 1, 128)])
def test_flash_fwd_bwd(B, T, H, hd):
    torch.manual_seed(8)
    d = H * hd
    qkv = _rand(B * T, 3 * d, scale=1.0)
    out = torch.zeros(B * T, d, device=DEV, dtype=torch.bfloat16)
    lse = torch.zeros(B, H, T, device=DEV)
    ops.flash_fwd(qkv, out, lse, B, T, H, hd)
    out2 = torch.empty_like(out); lse2 = torch.empty_like(lse)
    ref.flash_fwd(qkv, out2, lse2, B, T, H, hd)
    torch.cuda.synchronize()
    assert ops.error_word() == 0
    assert relerr(out, out2) < 1e-2, relerr(out, out2)
    assert relerr(lse, lse2) < 1e-3
    dout = _rand(B * T, d)
    dqkv = torch.zeros_like(qkv); delta = torch.empty(B, H, T, device=DEV)
    ops.flash_bwd(qkv, out, dout, lse, dqkv, delta, B, T, H, hd)
    dqkv2 = torch.zeros_like(qkv)
    ref.flash_bwd(qkv, out2, dout, lse2, dqkv2, B, T, H, hd)
    torch.cuda.synchronize()
    assert ops.error_word() == 0
    for i, name in enumerate("qkv"):
        e = relerr(dqkv[:, i * d:(i + 1) * d], dqkv2[:, i * d:(i + 1) * d])
        assert e < 2e-2, (name, e)
    # every output element has one writer and a fixed summation order: identical bits on a second run
    out3, lse3, dqkv3 = torch.zeros_like(out), torch.zeros_like(lse), torch.zeros_like(dqkv)
    ops.flash_fwd(qkv, out3, lse3, B, T, H, hd)
    ops.flash_bwd(qkv, out, dout, lse, dqkv3, delta, B, T, H, hd)
    assert torch.equal(out, out3) and torch.equal(lse, lse3) and torch.equal(dqkv, dqkv3)


@pytest.mark.parametrize("B,T,H,hd", [(74, 64, 8, 128), (75, 64, 8, 128), (55, 49, 8, 128), (56, 49, 8, 128), (185, 48, 8, 128),
                                      (186, 48, 8, 128), (259, 40, 8, 128), (260, 33, 8, 128), (74, 128, 8, 128), (75, 128, 8, 128),
                                      (80, 65, 16, 128)])
def test_flash_short_sequences_of_many_items(B, T, H, hd):
    """Up to 128 positions at head width 128 and many items: the kernel for short sequences up to 64 positions, beyond them the 128-row
    tiles with one tile per item, on both sides of the line at which the backward kernel for those comes in."""
    test_flash_fwd_bwd(B, T, H, hd)


@pytest.mark.parametrize("B,T,H,hd", [(32, 256, 8, 64), (40, 130, 8, 64), (3, 1777, 4, 64), (75, 72, 2, 64), (74, 72, 2, 64)])
def test_flash_backward_with_two_ctas_per_sm(B, T, H, hd):
    """Head width 64 with more (batch, head, tile) items than SMs: two CTAs share an SM, with one S / dP buffer and a two-stage ring
    each.  Up to several items a CTA (the barrier phases carry over), ragged lengths; the last shape is one item below the line."""
    test_flash_fwd_bwd(B, T, H, hd)


@pytest.mark.parametrize("B,T,H,hd", [(1, 200, 150, 64), (2, 129, 160, 64), (1, 385, 151, 64), (2, 257, 50, 128), (3, 130, 74, 128)])
def test_flash_items_handed_out_there_and_back(B, T, H, hd):
    """Items of unequal length in two to five rounds over the CTAs, odd rounds from the last CTA to the first, the last round with a few
    items, one short of full and exactly full (148 CTAs, 296 where two share an SM); warps all of whose keys come after their queries."""
    test_flash_fwd_bwd(B, T, H, hd)


@pytest.mark.parametrize("B,T,H,hd", [(1, 200, 2, 64), (4, 200, 80, 64), (1, 200, 2, 128), (2, 50, 2, 64)])
@pytest.mark.parametrize("bad", [float("nan"), 3e38])
def test_flash_backward_of_a_query_without_a_softmax(B, T, H, hd, bad):
    """A query whose scores are NaN, or all -inf, has no softmax and no gradient, but the keys after it do not see it: their dV has the bits of
    a call without that query's fault, in the tile of the diagonal too."""
    torch.manual_seed(T + hd)
    d, at = H * hd, 37
    qkv, dout = _rand(B * T, 3 * d), _rand(B * T, d)
    dv = []
    for value in (None, bad):
        x = qkv.clone()
        x[:, d:2 * d] = x[:, d:2 * d].abs() + 0.1            # positive keys: a query of -3e38 scores -inf everywhere
        if value is not None:
            x[at, :d] = -value                               # in the first sequence
        out, lse, delta, dqkv = torch.empty(B * T, d, device=DEV).bfloat16(), torch.empty(B, H, T, device=DEV), torch.empty(B, H, T, device=DEV), torch.empty_like(x)
        ops.flash_fwd(x, out, lse, B, T, H, hd)
        ops.flash_bwd(x, out, dout, lse, dqkv, delta, B, T, H, hd)
        assert value is None or out[at].isnan().all()
        dv.append(dqkv[:, 2 * d:])
    assert dv[1][:at + 1].isnan().all() and torch.equal(dv[0][at + 1:], dv[1][at + 1:]) and not dv[0].isnan().any()


def test_flash_large_scores_rescale():
    """Scores that keep growing along the keys force the in-place rescaling of the output accumulator."""
    torch.manual_seed(21)
    B, T, H, hd = 1, 512, 2, 128
    d = H * hd
    qkv = _rand(B * T, 3 * d, scale=1.0)
    ramp = torch.linspace(0.2, 6.0, T, device=DEV)[:, None]
    qkv[:, d:2 * d] = (qkv[:, d:2 * d].float() * ramp).bfloat16()      # later keys have larger norms
    out = torch.zeros(B * T, d, device=DEV, dtype=torch.bfloat16)
    lse = torch.zeros(B, H, T, device=DEV)
    ops.flash_fwd(qkv, out, lse, B, T, H, hd)
    out2 = torch.empty_like(out); lse2 = torch.empty_like(lse)
    ref.flash_fwd(qkv, out2, lse2, B, T, H, hd)
    torch.cuda.synchronize()
    assert ops.error_word() == 0
    assert relerr(out, out2) < 1e-2, relerr(out, out2)
    assert relerr(lse, lse2) < 1e-3


@pytest.mark.parametrize("M", [1, 8, 17, 32, 64])
@pytest.mark.parametrize("N,K", [(3072, 1024), (1024, 4096), (50257, 1024), (200, 192)])
def test_gemm_skinny(M, N, K):
    torch.manual_seed(9)
    x = _rand(M, K, scale=0.5)
    w = _rand(N, K, scale=0.1)
    bias = _rand(N)
    ld = (N + 63) // 64 * 64
    scratch = torch.zeros(ops.gemm_skinny_scratch_elems(M, N, K), device=DEV)
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID):
        aux = _rand(M, ld)[:, :N]
        aux_ref = aux.clone()
        out = torch.zeros(M, ld, device=DEV, dtype=torch.bfloat16)[:, :N]
        want = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
        ops.gemm_skinny(x, w, out, scratch, epi=epi, bias=bias, aux=aux)
        ref.gemm(x, w, want, False, False, False, epi, bias, aux_ref, 1.0)
        assert relerr(out, want) < 8e-3, (epi, relerr(out, want))
        out2 = torch.zeros_like(out)
        ops.gemm_skinny(x, w, out2, scratch, epi=epi, bias=bias, aux=aux_ref.clone())
        assert torch.equal(out, out2)               # split-K partials are added in a fixed order
    torch.cuda.synchronize()
    assert ops.error_word() == 0


@pytest.mark.parametrize("M", [1, 5, 16])
@pytest.mark.parametrize("N,K", [(3072, 1024), (4096, 1024), (50257, 1024), (200, 192)])
def test_gemm_skinny_with_layernorm_prologue(M, N, K):
    """LayerNorm folded into the weight-streaming GEMM equals LayerNorm followed by the GEMM."""
    torch.manual_seed(10)
    x = _rand(M, K, scale=2.0) + 0.5
    w = _rand(N, K, scale=0.1)
    bias = _rand(N)
    lw, lb = (1.0 + 0.1 * torch.randn(K, device=DEV)).bfloat16(), (0.1 * torch.randn(K, device=DEV)).bfloat16()
    ld = (N + 63) // 64 * 64
    scratch = torch.zeros(ops.gemm_skinny_scratch_elems(M, N, K), device=DEV)
    y = torch.empty_like(x)
    ref.layernorm_fwd(x, lw, lb, y, None, None)
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_BIAS_GELU):
        aux = torch.zeros(M, ld, device=DEV, dtype=torch.bfloat16)[:, :N]
        aux_ref = aux.clone()
        out = torch.zeros(M, ld, device=DEV, dtype=torch.bfloat16)[:, :N]
        want = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
        ops.gemm_skinny(x, w, out, scratch, epi=epi, bias=bias, aux=aux, ln_w=lw, ln_b=lb)
        ref.gemm(y, w, want, False, False, False, epi, bias, aux_ref, 1.0)
        assert relerr(out, want) < 1e-2, (epi, relerr(out, want))
    torch.cuda.synchronize()
    assert ops.error_word() == 0


def test_tensor_map_cache_overflow_keeps_descriptors_valid():
    """The descriptor cache drops its index when full; descriptors handed out before (the A map of
    the very launch whose B map caused the overflow) must stay valid, so results stay right."""
    from kharon_b200 import _native
    lib = _native.cuda()
    old = lib.kh_tmap_cache_limit(7)
    try:
        torch.manual_seed(11)
        big_a = _rand(128 + 400, 192, scale=0.5)
        big_b = _rand(256 + 400, 192, scale=0.2)
        out = torch.empty(128, 256, device=DEV, dtype=torch.bfloat16)
        want = torch.empty_like(out)
        for i in range(0, 400, 3):          # every launch sees operands at new addresses
            a, b = big_a[i:i + 128], big_b[i + 1:i + 257]
            ops.gemm(a, b, out)
            ref.gemm(a, b, want, False, False, False, ops.EPI_NONE, None, None, 1.0)
            assert relerr(out, want) < 8e-3, i
    finally:
        lib.kh_tmap_cache_limit(old)
    torch.cuda.synchronize()
    assert ops.error_word() == 0


def test_bounded_wait_status_word_is_clean():
    assert ops.error_word() == 0


def test_bounded_wait_runs_out_and_reports_status():
    """A wait on a flag that nothing sets gives up after its limit, reports code 5 through the status
    word, and leaves the context usable; once the flag is set the same wait succeeds."""
    flag = torch.zeros(1, device=DEV, dtype=torch.int32)
    status = torch.full((1,), -1, device=DEV, dtype=torch.int32)
    ops.wait_probe(flag, 1, 30, status)
    torch.cuda.synchronize()
    assert status.item() == 5 and ops.error_word() == 5      # read-and-clear
    assert ops.error_word() == 0
    flag.fill_(1)
    ops.wait_probe(flag, 1, 30, status)
    torch.cuda.synchronize()
    assert status.item() == 0 and ops.error_word() == 0
    assert torch.ones(4, device=DEV).sum().item() == 4.0     # the context still works


def test_mailbox_put_then_wait_and_wait_that_runs_out():
    """The pipeline mailbox primitives on one device (the slot is local memory here): a put delivers
    the bytes and raises the slot counter, the wait queued behind it passes and advances its expected
    count; a wait for a message nobody sends gives up after its limit with code 7."""
    src = _rand(300, 64)
    dst = torch.zeros_like(src)
    flag = torch.zeros(1, device=DEV, dtype=torch.int32)
    state = torch.zeros(2, device=DEV, dtype=torch.int32)
    expected = torch.zeros(1, device=DEV, dtype=torch.int32)
    for k in range(1, 4):
        src.add_(1.0)
        ops.p2p_put(src, dst.data_ptr(), flag.data_ptr(), state)
        ops.p2p_wait(flag.data_ptr(), expected, 500)
        torch.cuda.synchronize()
        assert torch.equal(dst, src) and flag.item() == k and expected.item() == k
        assert state.tolist() == [k, 0] and ops.error_word() == 0
    ops.p2p_wait(flag.data_ptr(), expected, 50)          # message 4 never comes
    torch.cuda.synchronize()
    assert ops.error_word() == 7 and expected.item() == 3
    assert ops.error_word() == 0


def test_guard_bands_stay_intact_through_training_steps():
    from kharon_b200.engine import TrainEngine
    from kharon_b200.models import gpt
    from kharon_b200.utils.guards import GuardedAlloc
    from kharon_b200.utils.rng import Rng
    ga = GuardedAlloc()
    gpt.set_allocator(ga)
    try:
        e = TrainEngine(layers=2, d_model=128, heads=2, vocab=1000, seq=96, mbatch=3, n_micro=2, device="cuda")
    finally:
        gpt.set_allocator(None)
    idx, tgt = Rng(4).batch(e.tokens_per_step, 1000)
    for _ in range(3):
        e.train_step(idx, tgt)
    torch.cuda.synchronize()
    assert len(ga.bufs) > 20 and ga.check() == []
    ga.bufs[0][1][3] = 0          # a damaged band is reported
    assert ga.check() == [ga.bufs[0][0]]


def test_merge_attention_equals_attention_over_all_keys():
    torch.manual_seed(11)
    H, T, hd = 2, 64, 64
    q, k, v = (torch.randn(H, T, hd, device=DEV) for _ in range(3))
    def attn(kk, vv):
        s = (q @ kk.transpose(-1, -2)) / hd ** 0.5
        return torch.softmax(s, -1) @ vv, torch.logsumexp(s, -1)
    o_all, l_all = attn(k, v)
    o1, l1 = attn(k[:, :40], v[:, :40])
    o2, l2 = attn(k[:, 40:], v[:, 40:])
    o, l = ops.merge_attention(o1, l1, o2, l2)
    assert torch.allclose(o, o_all, atol=1e-5) and torch.allclose(l, l_all, atol=1e-5)


def test_grpo_device_advantages_and_coefficients_match_host():
    """Device versions of the group-relative advantages and the per-token GRPO coefficients against the
    runtime library's host functions (reference src/core/grpo.c:7-20, src/grpo_train.c:164-174)."""
    torch.manual_seed(30)
    NP, G, T = 6, 8, 18
    rows = NP * G
    rew = torch.rand(rows)
    rew[8:16] = 0.5                                   # a group with zero variance
    p_cur, p_ref = torch.rand(rows * T) * 0.9 + 1e-3, torch.rand(rows * T) * 0.9 + 1e-3
    adv_h, coef_h = torch.empty(rows), torch.empty(rows * T)
    ops.grpo_advantages(rew, NP, G, 1e-4, adv_h)
    ops.grpo_coef(adv_h, p_cur, p_ref, rows, T, 8, T - 2, 0.04, coef_h)
    adv_d, coef_d = torch.empty(rows, device=DEV), torch.empty(rows * T, device=DEV)
    ops.grpo_advantages(rew.to(DEV), NP, G, 1e-4, adv_d)
    ops.grpo_coef(adv_d, p_cur.to(DEV), p_ref.to(DEV), rows, T, 8, T - 2, 0.04, coef_d)
    assert torch.allclose(adv_d.cpu(), adv_h, rtol=1e-5, atol=1e-6)
    assert torch.allclose(coef_d.cpu(), coef_h, rtol=1e-4, atol=1e-7)


@pytest.mark.parametrize("hd,H,lens", [(64, 4, [1]), (64, 2, [129, 64, 1, 300, 128, 2]), (128, 3, [65, 511, 127]),
                                       (64, 1, [40 + 17 * i for i in range(19)]), (64, 1, [1000 * 66, 5])])
def test_flash_varlen_matches_one_launch_per_sequence(hd, H, lens):
    """Several sequences in one launch against the single-sequence launch of the same kernel, which does the same arithmetic
    tile by tile: identical bits.  Rows between the sequences hold NaN and must neither be read into a result nor written;
    more sequences than one launch holds; a sequence with more query tiles than the list of pairs."""
    torch.manual_seed(len(lens))
    rows = sum(lens) + 3 * len(lens)
    qkv = torch.full((rows, 3 * H * hd), float("nan"), device="cuda").bfloat16()
    segs, r = [], 2
    for n in lens:
        segs.append((r, n))
        qkv[r:r + n] = torch.randn(n, 3 * H * hd, device="cuda").bfloat16()
        r += n + 3
    out = torch.full((rows, H * hd), 7.0, device="cuda").bfloat16()
    want = out.clone()
    lse = torch.empty(H * max(lens), device="cuda")
    for r, n in segs:
        if n > 64:
            ops.flash_fwd(qkv[r:r + n], want[r:r + n], lse, 1, n, H, hd)
        else:                                            # (short sequences by themselves take another kernel)
            ops.flash_fwd_varlen(qkv[r:r + n], want[r:r + n], [(0, n)], H, hd)
            ref.flash_fwd(qkv[r:r + n].float(), out[r:r + n], None, 1, n, H, hd)
            assert relerr(want[r:r + n], out[r:r + n]) < 1e-2
            out[r:r + n] = 7.0
    ops.flash_fwd_varlen(qkv, out, segs, H, hd)
    assert torch.equal(out, want) and not out.isnan().any()
    assert ops.error_word() == 0


@pytest.mark.parametrize("B,T,H,hd", [(1, 1, 1, 64), (3, 5, 2, 64), (40, 18, 8, 64), (2, 16, 3, 128), (5, 33, 2, 128), (4, 48, 4, 64), (2, 64, 3, 64),
                                      (2, 64, 2, 128)])
def test_flash_short_sequences(B, T, H, hd):
    """Attention of up to 64 positions (its own kernels) against fp64: P and dS round to bf16 (2^-9 each), outputs once more;
    the tile kernels, measured the same way, are off by 2.4e-3."""
    torch.manual_seed(B + T)
    d = H * hd
    qkv, dout = torch.randn(B * T, 3 * d, device="cuda").bfloat16(), torch.randn(B * T, d, device="cuda").bfloat16()
    out, lse = torch.empty(B * T, d, device="cuda", dtype=torch.bfloat16), torch.empty(B, H, T, device="cuda")
    dqkv, delta = torch.full_like(qkv, 7.0), torch.empty(B, H, T, device="cuda")
    ops.flash_fwd(qkv, out, lse, B, T, H, hd)
    ops.flash_bwd(qkv, out, dout, lse, dqkv, delta, B, T, H, hd)
    x = qkv.double().requires_grad_()
    q, k, v = x.view(B, T, 3, H, hd).permute(2, 0, 3, 1, 4)
    s = (q @ k.transpose(-1, -2)) / hd ** 0.5
    s = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    o = (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3).reshape(B * T, d)
    o.backward(dout.double())
    assert relerr(out, o) < 4e-3 and relerr(lse, torch.logsumexp(s, -1)) < 1e-5
    assert relerr(dqkv, x.grad) < (6e-3 if T > 1 else 1e-2)
    again = torch.empty_like(dqkv)
    ops.flash_bwd(qkv, out, dout, lse, again, delta, B, T, H, hd)
    assert torch.equal(again, dqkv) and ops.error_word() == 0


@pytest.mark.parametrize("rows,V,d", [(1, 3, 64), (257, 2, 64), (1000, 9, 130), (2049, 700, 256)])
def test_embedding_gradient_with_repeated_ids(rows, V, d):
    """Ids that occur 1 to 500 times (the list of later rows holds 64), rows around the scan's turns of 256: fp32 sums in row order,
    the order of the reference loop, so the bits agree."""
    g = torch.Generator().manual_seed(rows)
    tok = torch.randint(0, V, (rows,), generator=g)
    tok[: min(rows, 66)] = 0
    dx = torch.randn(rows, d, generator=g).bfloat16()
    want = torch.zeros(V, d)
    for i in range(rows):
        want[tok[i]] += dx[i].float()
    dwte = torch.zeros(V, d, device="cuda")
    ops.embed_bwd(tok.int().cuda(), dx.cuda(), dwte, None, 1, rows)
    assert torch.equal(dwte.cpu(), want)


@pytest.mark.parametrize("later", [1, 7, 63, 64, 65, 127, 128, 129, 300, 1000])
def test_embedding_gradient_of_an_id_with_many_later_rows(later):
    """One id with exactly so many later rows (a list holds 64), close together and far apart, over three column chunks: the order of
    the reference loop, so the bits agree."""
    g = torch.Generator().manual_seed(later)
    for rows in (later + 1, later + 300, 3 * later + 700):
        tok = torch.full((rows,), 1)
        at = torch.randperm(rows, generator=g)[:later + 1]
        tok[at] = 0
        tok[(tok == 1).nonzero().flatten()[::2]] = 2
        dx = torch.randn(rows, 514, generator=g).bfloat16()
        want = torch.zeros(3, 514)
        for i in range(rows):
            want[tok[i]] += dx[i].float()
        dwte = torch.zeros(3, 514, device="cuda")
        ops.embed_bwd(tok.int().cuda(), dx.cuda(), dwte, None, 1, rows)
        assert torch.equal(dwte.cpu(), want), rows


@pytest.mark.parametrize("M,N,K,blk", [(1, 328, 64, 0), (9, 4096, 1024, 0), (130, 1000, 72, 64), (300, 520, 2048, 0), (257, 768, 512, 128), (2200, 4096, 1024, 512),
                                       (700, 1016, 256, 4096 * 2 + 64)])
def test_gemm_gelu_without_the_pre_activation(M, N, K, blk):
    """Bias + GELU without its pre-activation gives the same bits as with it: every kernel of the family, ragged edges."""
    torch.manual_seed(M)
    a, b, bias, aux = _rand(M, K, scale=0.5), _rand(N, K, scale=0.1), _rand(N), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    want, out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, want, epi=ops.EPI_BIAS_GELU, bias=bias, aux=aux, block_n=blk)
    ops.gemm(a, b, out, epi=ops.EPI_GELU, bias=bias, block_n=blk)
    assert torch.equal(out, want)
    if M <= ops.SKINNY_MAX_ROWS:
        scratch = torch.zeros(ops.gemm_skinny_scratch_elems(M, N, K), device=DEV)
        ops.gemm_skinny(a, b, want, scratch, epi=ops.EPI_BIAS_GELU, bias=bias, aux=aux)
        ops.gemm_skinny(a, b, out, scratch, epi=ops.EPI_GELU, bias=bias)
        assert torch.equal(out, want)
    assert ops.error_word() == 0


@pytest.mark.parametrize("rows,d", [(1, 8), (3, 128), (31, 264), (33, 512), (4737, 520), (1000, 1024), (5, 1032), (2400, 2040), (700, 2048), (9, 4096), (600, 3080), (70, 4104)])
def test_layernorm_backward_against_fp64(rows, d):
    """Ragged rows and widths on both sides of 512, 1024, 2048 and 4096 columns (one to eight warps per row, the two kernels beyond), with and
    without the residual gradient: column sums to fp32 rounding (n additions of terms below 8: 1e-5 of their norm), dx to bf16 rounding."""
    torch.manual_seed(rows + d)
    x, w, dy, dres = _rand(rows, d), _rand(d), _rand(rows, d), _rand(rows, d)
    X, G = x.double(), dy.double()
    mean, rstd = X.mean(1).float(), (X.var(1, unbiased=False) + 1e-5).rsqrt().float()
    xh = (X - mean.double()[:, None]) * rstd.double()[:, None]
    g = G * w.double()
    base = rstd.double()[:, None] * (g - g.mean(1, keepdim=True) - xh * (g * xh).mean(1, keepdim=True))
    for res in (dres, None):
        dx = torch.full((rows + 1, d), 7.0, device=DEV, dtype=torch.bfloat16)
        dw, db = torch.ones(d, device=DEV), torch.full((d,), 2.0, device=DEV)
        part = torch.zeros(ops.layernorm_bwd_scratch_elems(rows, d), device=DEV)
        for k in (1, 2):               # the scratch is ready for another call
            ops.layernorm_bwd(dy, x, w, mean, rstd, res, dx[:rows], dw, db, part)
            want = base + (res.double() if res is not None else 0)
            assert ((dx[:rows].double() - want).norm() / want.norm()).item() < 2.0 ** -8
            for got, one, sums in ((dw, 1.0, (G * xh).sum(0)), (db, 2.0, G.sum(0))):
                assert ((got.double() - one - k * sums).norm() / (k * sums.norm() + one)).item() < 1e-5
        assert (dx[rows] == 7).all()
    again = torch.ones(d, device=DEV)
    ops.layernorm_bwd(dy, x, w, mean, rstd, dres, dx[:rows], again, db, part)
    once = torch.ones(d, device=DEV)
    ops.layernorm_bwd(dy, x, w, mean, rstd, dres, dx[:rows], once, db, part)
    assert torch.equal(again, once) and ops.error_word() == 0


@pytest.mark.parametrize("split", [2, 3, 4])
@pytest.mark.parametrize("M,N,K", [(256, 256, 1024), (264, 248, 600), (8, 520, 1000), (1000, 136, 4096), (1536, 512, 900)])
def test_gemm_split_k_on_cta_pairs(M, N, K, split):
    """256 x 256 tiles of CTA pairs whose K is shared by two to four pairs of a cluster: edges of the tiles, a last slice that is shorter, every
    operand order, column sums and epilogues, against fp64 and against the form without a split."""
    torch.manual_seed(M + N + K + split)
    if (split - 1) * -(-(-(-K // 64)) // split) >= -(-K // 64):
        pytest.skip("a slice would be empty")
    pad = lambda n: (n + 7) // 8 * 8
    r = lambda *s: _rand(*s, scale=0.5)
    blk = 4096 * split + 512
    for a_mn, b_mn in ((1, 1), (0, 0), (0, 1), (1, 0)):
        a, b = (r(K, pad(M))[:, :M] if a_mn else r(M, pad(K))[:, :K]), (r(K, pad(N))[:, :N] if b_mn else r(N, pad(K))[:, :K])
        want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
        big = torch.full((M + 1, pad(N)), 3.0, device=DEV)
        db = torch.ones(M, device=DEV) if a_mn else None
        ops.gemm(a, b, big[:M, :N], a_mn=bool(a_mn), b_mn=bool(b_mn), accumulate=True, colsum=db, block_n=blk)
        assert ((big[:M, :N].double() - 3 - want).norm() / want.norm()).item() < 1e-5
        assert (big[M] == 3).all() and (big[:, N:] == 3).all()
        if a_mn:
            cs = a.double().sum(0)
            assert ((db.double() - 1 - cs).norm() / cs.norm()).item() < 2e-4
        again = torch.full((M, pad(N)), 3.0, device=DEV)
        ops.gemm(a, b, again[:, :N], a_mn=bool(a_mn), b_mn=bool(b_mn), accumulate=True, colsum=db, block_n=blk)
        assert torch.equal(again, big[:M])
    bias, res = r(pad(N))[:N], r(M, pad(N))[:, :N]
    a, b = r(M, pad(K))[:, :K], r(N, pad(K))[:, :K]
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_BIAS_GELU, ops.EPI_BIAS_RESID, ops.EPI_DGELU, ops.EPI_RESID, ops.EPI_GELU):
        out = {}
        for w in (blk, 512):
            o, aux = torch.full((M, pad(N)), 7.0, device=DEV).bfloat16(), res.clone().contiguous() if N % 8 == 0 else torch.zeros(M, pad(N), device=DEV).bfloat16()[:, :N].copy_(res)
            ops.gemm(a, b, o[:, :N], epi=epi, bias=bias if epi in (1, 2, 3, 6) else None, aux=aux if epi in (2, 3, 4, 5) else None, block_n=w)
            out[w] = o
        x, y = out[blk].double(), out[512].double()
        assert ((x - y).norm() / y.norm()).item() < 2.0 ** -8 and torch.equal(out[blk][:, N:], out[512][:, N:])
    assert ops.error_word() == 0


def test_layernorm_backward_takes_any_scratch():
    """A scratch that starts on any fp32 element serves (off 16 bytes by the two kernels of wide rows: 1e-5 for another order of the sums, a bf16 step for
    dx), and its counters stay zero."""
    torch.manual_seed(3)
    for rows, d in ((300, 264), (300, 1024), (130, 2048), (40, 4096)):
        x, w, dy = _rand(rows, d), _rand(d), _rand(rows, d)
        mean, rstd = x.float().mean(1), (x.float().var(1, unbiased=False) + 1e-5).rsqrt()
        n = ops.layernorm_bwd_scratch_elems(rows, d)
        out = []
        for off in (0, 1, 2):
            part = torch.zeros(n + off, device=DEV)[off:]
            dx, dw, db = torch.empty_like(x), torch.zeros(d, device=DEV), torch.zeros(d, device=DEV)
            ops.layernorm_bwd(dy, x, w, mean, rstd, None, dx, dw, db, part)
            out.append((dx, dw, db))
            assert off == 0 or not part[:1024].any()
        for o in out[1:]:
            assert all(relerr(a, b) < t for a, b, t in zip(o, out[0], (2.0 ** -8, 1e-5, 1e-5)))


@pytest.mark.parametrize("d", [256, 4096, 4104])
def test_layernorm_backward_refuses_an_empty_problem(d):
    x, v = torch.zeros(1, d, device=DEV).bfloat16(), torch.zeros(d, device=DEV)
    part = torch.zeros(ops.layernorm_bwd_scratch_elems(1, d), device=DEV)
    with pytest.raises(ops.KernelError):
        ops.layernorm_bwd(x[:0], x[:0], x[0], v, v, None, x[:0], v, v, part)
