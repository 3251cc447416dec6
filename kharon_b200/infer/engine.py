"""Paged-KV inference engine: continuous batching, copy-on-write prefix sharing, on-device
sampling, CUDA-graph decode steps.

Division of labour:

* native scheduler (csrc/runtime/kharon_rt.cpp, ``kh_eng_*``): reference-counted block pool
  with a LIFO free list, per-sequence block tables, admission of waiting sequences, the flat
  token list of each mixed prefill+decode step, copy-on-write of shared blocks, retirement;
* this module: device buffers, one packed host->device metadata copy per step, the forward
  pass on the native kernels, the sampler, one small device->host copy of the sampled ids.

Differences from the reference engine (src/core/infer.c): sampling runs on the GPU, so a step
moves ``n_seq`` ints to the host instead of ``n_seq x vocab`` logits (:183-195); block sharing
is reference-counted and lazy (a shared block is copied when a sequence first writes into
it) instead of an eager copy of the partial block at fork time (:315-387); decode steps of a
fixed batch size replay a captured CUDA graph; no fixed-size stack arrays (:231-233,280,323).
Accounting (tokens_decoded counts one token per active sequence per step, the prefill step
included) follows infer.c:295 so that tok/s is comparable.
"""
from __future__ import annotations

import ctypes as C
import os
import time

import numpy as np
import torch

from .. import _native, ops
from ..models import GPT


class InferStats(dict):
    pass


class InferEngine:
    def __init__(self, model: GPT, block_size=16, n_blocks=None, max_tokens=None, max_seqs=33, use_graphs=True,
                 persistent_decode=None, attn_splits=None, flash_prefill=True):
        cfg = model.cfg
        self.model, self.cfg = model, cfg
        self.dev, self.dt = model.device, model.dtype
        self.tp = model.tp
        self.bs = block_size
        self.max_lb = (cfg.seq + block_size - 1) // block_size
        self.max_seqs = max_seqs
        self.n_blocks = n_blocks if n_blocks is not None else max_seqs * self.max_lb + 16
        self.max_tokens = max_tokens if max_tokens is not None else max(cfg.seq, max_seqs) + 64
        self.Hl, self.hd = cfg.n_head // self.tp, cfg.head_dim
        lib = _native.rt()
        self._h = lib.kh_eng_create(self.bs, self.n_blocks, max_seqs, self.max_lb)
        if not self._h:
            raise _native.NativeError(lib.kh_last_error().decode())
        L, d, dl, fo = cfg.n_layer, cfg.d_model, cfg.d_model // self.tp, 4 * cfg.d_model // self.tp
        z = dict(device=self.dev)
        self.kc = torch.zeros(L, self.n_blocks, self.bs, self.Hl, self.hd, dtype=self.dt, **z)
        self.vc = torch.zeros_like(self.kc)
        # packed step metadata: tok | pos | slot | rows | btab | pairs
        mt, ms_ = self.max_tokens, max_seqs
        self._o_tok, self._o_pos, self._o_slot = 0, mt, 2 * mt
        self._o_rows = 3 * mt
        self._o_btab = 3 * mt + ms_
        self._o_pairs = self._o_btab + ms_ * self.max_lb
        self._o_step = self._o_pairs + 2 * ms_ * 4          # the step number: sampled steps replayed from a graph read it here
        self._n_meta = self._o_step + 4                      # {step number, seed low, seed high, unused}
        pin = self.dev.type == "cuda"
        self.h_meta = torch.zeros(self._n_meta, dtype=torch.int32, pin_memory=pin)
        self.np_meta = self.h_meta.numpy()            # the same memory: element writes without a tensor operation each
        self.h_seq_ids = torch.zeros(ms_, dtype=torch.int32)
        self._plan_n = (C.c_int32(), C.c_int32(), C.c_int32())
        base = self.h_meta.data_ptr()
        at = lambda o: base + 4 * o
        self._plan_args = (at(self._o_tok), at(self._o_pos), at(self._o_slot), at(self._o_rows), self.h_seq_ids.data_ptr(),
                           at(self._o_btab), C.byref(self._plan_n[0]), C.byref(self._plan_n[1]), at(self._o_pairs), ms_ * 4,
                           C.byref(self._plan_n[2]))
        self.d_meta = torch.zeros(self._n_meta, dtype=torch.int32, **z)
        v = lambda t, o, n: t[o:o + n]
        self.d_tok, self.d_pos, self.d_slot = v(self.d_meta, 0, mt), v(self.d_meta, mt, mt), v(self.d_meta, 2 * mt, mt)
        self.d_rows = v(self.d_meta, self._o_rows, ms_)
        self.d_btab = v(self.d_meta, self._o_btab, ms_ * self.max_lb).view(ms_, self.max_lb)
        self.d_pairs = v(self.d_meta, self._o_pairs, 2 * ms_ * 4)
        self.d_stepno = v(self.d_meta, self._o_step, 3)
        e = lambda *s: torch.empty(*s, dtype=self.dt, **z)
        self.x = [e(mt, d), e(mt, d)]
        self.xmid, self.ln, self.qkv, self.att = e(mt, d), e(mt, d), e(mt, 3 * dl), e(mt, dl)
        self.act = e(mt, fo)
        self.last = e(ms_, d)
        self.lnf = e(ms_, d)
        self.logits = torch.zeros(ms_, model.Vp, dtype=self.dt, **z)
        self.d_out = torch.zeros(ms_ * 64, dtype=torch.int32, **z)
        self.h_out = torch.zeros(ms_ * 64, dtype=torch.int32, pin_memory=pin)
        # bf16 engines on a GPU sample up to this many ids straight into pinned memory: no copy back behind the step (us a step of a whole
        # generate call, L4 d256, copied / straight: 1 id 102.0 / 92.6, 8 114.8 / 109.0, 16 129.5 / 123.8, 32 180.0 / 169.5, 64 199.0 / 194.9; from 96 on the bus
        # takes as long as the copy: 96 227.1 / 226.4, 128 250.8 / 250.7, 256 341.2 / 341.4, 512 515.6 / 511.2)
        self._direct = 64 if pin and self.dt == torch.bfloat16 else 0
        # decode steps (few rows) use the weight-streaming split-K GEMM; its scratch covers every shape used
        self.skinny = None
        if self.dev.type == "cuda":
            shapes = [(3 * dl, d), (d, dl), (fo, d), (d, fo), (cfg.vocab, d)]
            n = max(ops.gemm_skinny_scratch_elems(ops.SKINNY_MAX_ROWS, N, K) for N, K in shapes)
            self.skinny = torch.zeros(n, dtype=torch.float32, **z)
        # Decode steps of up to ``persistent_max`` sequences run all layers and the head in one persistent kernel
        # when the shape allows it (ops.decode_layers); KHARON_PERSISTENT_DECODE=0 or persistent_decode=False keeps
        # the five-kernel chain.  The limit by width is measured (us a step, persistent / chain):
        #   L24 d1024, context 200: G = 8 415 / 1660, 16 573 / 1894, 17 773 / 1063, 24 873 / 1087, 32 936 / 1135; context 900: G = 17 1231 /
        #   1436, 32 1811 / 1721;
        #   L24 d1280: G = 16 1139 / 2095, 17 1664 / 1219, 32 2083 / 1436 (the chain's tensor-core GEMM starts at 17 rows);
        #   L24 d2048, context 300: G = 16 1537 / 3459, 17 2478 / 1832 (two launches), 32 3080 / 1933.
        if persistent_decode is None:
            persistent_decode = os.environ.get("KHARON_PERSISTENT_DECODE", "1") != "0"
        self.persistent = bool(persistent_decode and self.skinny is not None and self.tp == 1 and self.dt == torch.bfloat16
                               and ops.decode_layers_ok(1, d, cfg.n_head, cfg.head_dim, cfg.seq))
        self.persistent_max, self.skinny_rows = 0, ops.SKINNY_BEST_ROWS
        if self.persistent:
            rows = ops.decode_layers_rows(d)
            self.persistent_max = int(os.environ.get("KHARON_PERSISTENT_MAX_G", rows if d <= 1024 else min(16, rows)))
            # Widths of which one launch holds eight (3584 and more): steps of 9 to 16 rows take the chain with the tensor-core GEMM
            # (d4096, 16 rows, qkv / proj / fc / fcproj / head: 22 / 10 / 30 / 29 / 79 us; skinny 48 / 28 / 59 / 132 / 113).
            self.skinny_rows = min(self.skinny_rows, rows)
            names = ("ln1_w", "ln1_b", "qkv_w", "qkv_b", "proj_w", "proj_b", "ln2_w", "ln2_b", "fc_w", "fc_b",
                     "fcproj_w", "fcproj_b")
            self.layer_table = torch.tensor([[model.L(l, n).data_ptr() for n in names] for l in range(L)],
                                            dtype=torch.int64, device=self.dev)
            self.decode_work = ops.decode_layers_work(d, self.dev)
        # Contexts beyond 2048 positions: the keys of a token are cut into ranges with a CTA each (split-KV) and merged
        self.attn_splits = int(attn_splits) if attn_splits else (1 if cfg.seq <= 2048 else min(16, (cfg.seq + 2047) // 2048))
        self.attn_scratch = None
        if self.attn_splits > 1 and self.dev.type == "cuda":
            self.attn_scratch = torch.zeros(self.max_tokens * self.Hl * self.attn_splits * (self.hd + 1), dtype=torch.float32, **z)
        # Steps made of whole fresh prompts (every listed token belongs to a sequence that starts at position 0 in this
        # step) run their attention on the tensor cores with the training forward kernel, all prompts in one launch;
        # prompts beside decoding sequences, short and chunked ones go through the paged tile kernel (fp32 probabilities),
        # everything else through the paged kernel.
        self.flash_prefill = bool(flash_prefill and self.dev.type == "cuda" and self.dt == torch.bfloat16
                                  and self.hd in (64, 128))
        self._fresh = self._runs = None
        self._fused = False
        self.temperature, self.seed, self.step_no = 0.0, 0, 0
        # under TP the captured step contains the fused GEMM + all-reduce kernels (their call counter
        # is a device word); the NCCL seam is left to eager launches
        self.use_graphs = bool(use_graphs and self.dev.type == "cuda" and self.dt == torch.bfloat16
                               and (self.tp == 1 or getattr(model, "fused_tp", None) is not None))
        self.graphs = {}
        self._warm = set()
        self.d_step = None
        self.launches = 0

    def close(self):
        if self._h:
            _native.rt().kh_eng_free(self._h)
            self._h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def set_sampling(self, temperature: float, seed: int):
        """temperature <= 0: greedy.  Otherwise categorical draws seeded by (seed, step, row)."""
        self.temperature, self.seed = float(temperature), int(seed)       # (captured steps are keyed by the temperature;
                                                                          #  seed and step number travel in d_meta)

    def set_eos(self, eos: int):
        _native.rt().kh_eng_set_eos(self._h, eos)

    # ------------------------------------------------------------------ forward
    def _forward(self, ntok, nseq, rep=1):
        m, cfg = self.model, self.cfg
        P = m.params.c
        x, nxt = self.x
        tok, pos, slot = self.d_tok[:ntok], self.d_pos[:ntok], self.d_slot[:ntok]
        xs = x[:ntok]
        ops.embed_fwd(tok, pos, P["wte"], P["wpe"], xs, cfg.seq)
        if self._fused:       # layers and head in one kernel; only the sampler follows
            ops.decode_layers(xs, None, None, None, None, self.layer_table,
                              cfg.n_layer, self.Hl, self.hd, self.kc, self.vc, pos, slot, self.d_btab, self.bs, cfg.seq,
                              work=self.decode_work, head_w=m.head_weight(), lnf_w=P["lnf_w"], lnf_b=P["lnf_b"], logits=self.logits,
                              vocab=cfg.vocab, rows=self.d_rows, n_rows=nseq)
            ops.sample(self.logits, cfg.vocab, self.temperature, self.seed, self.step_no, rep, self.h_out if nseq * rep <= self._direct else self.d_out, nseq,
                       step_dev=self.d_stepno)
            return
        ln, qkv, att, xmid = self.ln[:ntok], self.qkv[:ntok], self.att[:ntok], self.xmid[:ntok]
        decode = ntok == nseq            # one new token per sequence: the attention kernel appends k, v itself
        if self._runs:
            runs = self._runs[0]
            rest = [(qkv[a:b], att[a:b], pos[a:b], slot[a:b]) for a, b in self._runs[1]]
        for l in range(cfg.n_layer):
            self._ln_lin(xs, m.L(l, "ln1_w"), m.L(l, "ln1_b"), ln, m.L(l, "qkv_w"), qkv, ops.EPI_BIAS, m.L(l, "qkv_b"))
            if not decode:
                ops.append_kv(qkv, self.kc[l], self.vc[l], pos, slot, self.d_btab, self.bs, self.Hl, self.hd, ntok)
            if not decode and self._fresh:
                ops.flash_fwd_varlen(qkv, att, self._fresh, self.Hl, self.hd)
            elif not decode and self._runs:
                ops.paged_prefill(qkv, self.kc[l], self.vc[l], att, pos, slot, self.d_btab, self.bs, self.Hl, self.hd, runs, cfg.seq)
                for q, o, p, s in rest:
                    ops.paged_attn(q, self.kc[l], self.vc[l], o, p, s, self.d_btab, self.bs, self.Hl, self.hd, q.shape[0], cfg.seq)
            else:
                ops.paged_attn(qkv, self.kc[l], self.vc[l], att, pos, slot, self.d_btab, self.bs, self.Hl, self.hd, ntok,
                               cfg.seq, append=decode, n_split=self.attn_splits, scratch=self.attn_scratch)
            # row-parallel products: one GEMM, or under TP the fused GEMM + all-reduce kernel / NCCL seam
            self._row(att, m.L(l, "proj_w"), xmid, m.L(l, "proj_b"), xs)
            self._ln_lin(xmid, m.L(l, "ln2_w"), m.L(l, "ln2_b"), ln, m.L(l, "fc_w"), self.act[:ntok], ops.EPI_GELU, m.L(l, "fc_b"))
            ys = nxt[:ntok]
            self._row(self.act[:ntok], m.L(l, "fcproj_w"), ys, m.L(l, "fcproj_b"), xmid)
            x, nxt = nxt, x
            xs = ys
        ops.gather_rows(xs, self.d_rows, self.last, nseq)
        self._ln_lin(self.last[:nseq], P["lnf_w"], P["lnf_b"], self.lnf[:nseq], m.head_weight(),
                     self.logits[:nseq, :cfg.vocab])
        ops.sample(self.logits, cfg.vocab, self.temperature, self.seed, self.step_no, rep, self.h_out if nseq * rep <= self._direct else self.d_out, nseq,
                       step_dev=self.d_stepno)

    def _lin(self, x, w, out, epi=ops.EPI_NONE, bias=None, aux=None):
        """Column-parallel / replicated linear layer: skinny kernel for decode-sized inputs."""
        if self.skinny is not None and x.shape[0] <= self.skinny_rows:
            ops.gemm_skinny(x, w, out, self.skinny, epi=epi, bias=bias, aux=aux, weights_static=True)
        else:
            ops.gemm(x, w, out, epi=epi, bias=bias, aux=aux)

    def _ln_lin(self, x, ln_w, ln_b, ln_out, w, out, epi=ops.EPI_NONE, bias=None, aux=None):
        """LayerNorm followed by a linear layer: for decode-sized inputs the skinny kernel normalises
        the rows itself (no LayerNorm launch, ``ln_out`` stays unused)."""
        if self.skinny is not None and x.shape[0] <= self.skinny_rows and x.shape[1] % 8 == 0:
            ops.gemm_skinny(x, w, out, self.skinny, epi=epi, bias=bias, aux=aux, ln_w=ln_w, ln_b=ln_b, weights_static=True)
        else:
            ops.layernorm_fwd(x, ln_w, ln_b, ln_out)
            self._lin(ln_out, w, out, epi, bias, aux)

    def _row(self, x, w, out, bias, resid):
        """Row-parallel linear layer (+ bias + residual); summed over the TP group when there is one."""
        if self.tp == 1:
            self._lin(x, w, out, ops.EPI_BIAS_RESID, bias, resid)
        else:
            self.model._row_parallel(x, w, out, bias, resid)

    def _fresh_prompts(self, ntok, nseq):
        """[(first row, length)] when every token of the step belongs to a prompt of at least 64 tokens that starts at position
        0 and is listed whole and contiguously; None otherwise (read from the host copy of the step's metadata).  A batch with
        a shorter prompt keeps the fp32 probabilities of the paged kernels: short prompts gain nothing from the 128-row tiles
        (16 heads of 64, 64 tokens: 3.9 us in the tile kernel, 4.4 here), longer ones beside them would (6 x 1000: 131 and 38)."""
        if not self.flash_prefill or ntok == nseq:
            return None
        pos = self.h_meta[self._o_pos:self._o_pos + ntok]
        slot = self.h_meta[self._o_slot:self._o_slot + ntok]
        cuts = [0] + (torch.nonzero(slot[1:] != slot[:-1]).flatten() + 1).tolist() + [ntok]
        out = []
        for a, b in zip(cuts[:-1], cuts[1:]):
            if int(pos[a]) != 0 or int(pos[b - 1]) != b - a - 1 or b - a < 64:
                return None
            out.append((a, b - a))
        return out if len(out) == nseq else None

    def _prompt_runs(self, ntok, nseq):
        """(runs, rest) of a step that lists several tokens of a sequence: runs = [(first row, length)] of at least sixteen
        consecutive positions of one sequence (shorter ones are faster a warp per token: nine-token prompts 1177 us a
        completion against 1224), rest = [(a, b)] the row ranges between them; None when there are no runs, when the tile
        kernel does not take the configuration, or when it would not earn its launch: beside the one for the rest while the
        step's (token, head) items are few (us, one launch / two, decoding sequences at 200 positions + prompt: H16 hd64, 8 + 16
        8.2 / 9.6, 8 + 48 10.1 / 9.9, 8 + 128 17.5 / 11.8, 31 + 24 12.4 / 12.3; H16 hd128, 31 + 32 18.3 / 19.5, 31 + 48 21.5 / 19.9;
        H8 hd32, 31 + 128 8.5 / 9.2, 31 + 4 x 64 10.7 / 8.2), and at head width 128 by itself (H16, 16 3.4 / 5.1, 48 7.5 / 5.9)."""
        if (ntok < nseq + 15 or self.dev.type != "cuda" or self.dt != torch.bfloat16 or self.attn_splits > 1
                or self.hd not in (32, 64, 128)):
            return None
        pos = self.np_meta[self._o_pos:self._o_pos + ntok]
        slot = self.np_meta[self._o_slot:self._o_slot + ntok]
        cuts = np.flatnonzero((slot[1:] != slot[:-1]) | (pos[1:] != pos[:-1] + 1)) + 1
        lo = np.concatenate(([0], cuts)).tolist()
        hi = lo[1:] + [ntok]
        runs, rest, at = [], [], 0
        for a, b in zip(lo, hi):
            if b - a >= 16:
                if at < a:
                    rest.append((at, a))
                runs.append((a, b - a))
                at = b
        if at < ntok:
            rest.append((at, ntok))
        least = {32: 1280, 64: 896, 128: 1100}[self.hd] if rest else 600 if self.hd == 128 else 1
        return (runs, rest) if runs and ntok * self.Hl >= least else None

    def _one_kernel(self, ntok, nseq):
        """Whether this step runs in the persistent kernel.  Over long contexts its W warps per (sequence, head) lose to the chain's
        attention (split-KV where the model has more than 2048 positions) once the sequences fill the SMs.  L4 d1024, 4200 positions, us a step, persistent / chain:
        sixteen heads, contexts 200 / 2000 / 3000 / 4000: G = 17 143 / 213, 319 / 437, 413 / 477, 511 / 501; 24 161 / 219, 436 / 480, 575 / 543, 715 / 571; 32 170 / 223,
        521 / 525, 701 / 621, 885 / 674; eight heads, 2000 / 3000 / 4000: 24 484 / 575, 652 / 636, 826 / 674; 32 501 / 639, 673 / 742, 848 / 791.  Context 8100 of
        16400: sixteen heads, G = 17 895 / 818, 24 1290 / 936; eight heads, 17 (136 items for 148 SMs) 849 / 960, 24 1527 / 1133."""
        if not (self.persistent and ntok == nseq and ntok <= self.persistent_max and ntok <= 32):
            return False
        return ntok <= 16 or ntok * self.Hl <= 148 or int(self.np_meta[self._o_pos:self._o_pos + ntok].max()) < (4096 if ntok <= 20 else 2560)

    def _run(self, ntok, nseq, rep=1):
        """Metadata is already in ``h_meta``; runs one step and returns the sampled ids (host)."""
        self._fused = self._one_kernel(ntok, nseq)
        self._fresh = self._fresh_prompts(ntok, nseq)
        self._runs = None if self._fresh else self._prompt_runs(ntok, nseq)
        sd = self.seed & 0xFFFFFFFFFFFFFFFF
        to_i32 = lambda u: u - (1 << 32) if u >= (1 << 31) else u
        self.np_meta[self._o_step:self._o_step + 3] = (self.step_no & 0x7FFFFFFF, to_i32(sd & 0xFFFFFFFF), to_i32(sd >> 32))
        key = (ntok, nseq, rep, self.temperature, self._fused)
        few = nseq * rep <= self._direct               # the copy of the metadata is part of a captured step (many: it starts earlier by itself)
        if self.use_graphs and ntok == nseq:           # greedy and sampled steps alike: the step number lives in d_meta
            g = self.graphs.get(key)
            if g is None and key in self._warm:
                torch.cuda.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    if few:
                        self.d_meta.copy_(self.h_meta, non_blocking=True)
                    self._forward(ntok, nseq, rep)
                self.graphs[key] = g
            if g is None or not few:
                self.d_meta.copy_(self.h_meta, non_blocking=True)
            if g is not None:
                g.replay()
            else:
                self._forward(ntok, nseq, rep)
                self._warm.add(key)
        else:
            self.d_meta.copy_(self.h_meta, non_blocking=True)
            self._forward(ntok, nseq, rep)
        self.step_no += 1
        n = nseq * rep
        if n > self._direct:
            self.h_out[:n].copy_(self.d_out[:n], non_blocking=True)
        if self.dev.type == "cuda":
            torch.cuda.current_stream().synchronize()
        return self.h_out[:n]

    # ------------------------------------------------------------------ scheduling
    def _plan(self, max_active):
        rc = _native.rt().kh_eng_plan(self._h, max_active, self.max_tokens, *self._plan_args)
        _native.rt_check(rc)
        return rc, self._plan_n[0].value, self._plan_n[1].value, self._plan_n[2].value

    def _step(self, max_active):
        rc, ntok, nseq, npairs = self._plan(max_active)
        if rc == 1 or nseq == 0:
            return False
        if npairs:
            self.d_meta.copy_(self.h_meta, non_blocking=True)
            ops.copy_blocks(self.kc, self.vc, self.d_pairs, npairs)
        out = self._run(ntok, nseq)
        _native.rt_check(_native.rt().kh_eng_commit(self._h, out.data_ptr(), nseq))
        return True

    def _stats(self):
        st = (C.c_int64 * 4)()
        _native.rt().kh_eng_stats(self._h, st)
        return InferStats(blocks_total=st[0], blocks_peak=st[1], tokens_decoded=st[2], prefix_blocks_saved=st[3])

    def _collect(self, sids):
        """Token lists of finished sequences, which are released."""
        lib, n = _native.rt(), len(sids)
        ids, lens = (C.c_int32 * n)(*sids), (C.c_int32 * n)()
        cap = sum(lib.kh_eng_seq_len(self._h, i) for i in sids) if n <= 4 else n * (self.max_lb * self.bs + 1)
        buf = (C.c_int32 * cap)()
        _native.rt_check(lib.kh_eng_collect(self._h, n, ids, buf, cap, lens))
        out, at = [], 0
        for k in lens:
            out.append(buf[at:at + k])
            at += k
        return out

    def _timer(self):
        if self.dev.type == "cuda":
            torch.cuda.synchronize()
        return time.perf_counter()

    def generate(self, prompts, n_new, max_active=None):
        """Independent generations with continuous batching: at most ``max_active`` sequences in
        flight, waiting ones are admitted as soon as a slot and blocks are free
        (infer_generate, src/core/infer.c:264-313).  Returns (token lists, stats, ms)."""
        lib = _native.rt()
        lib.kh_eng_reset(self._h)
        n = len(prompts)
        news = [n_new] * n if isinstance(n_new, int) else list(n_new)
        max_active = max_active or min(n, self.max_seqs)
        pending = list(range(n))
        sid_of = {}
        outs = [None] * n
        t0 = self._timer()
        while True:
            # feed the scheduler as sequence slots free up
            while pending:
                i = pending[0]
                p = torch.tensor(prompts[i], dtype=torch.int32)
                sid = lib.kh_eng_add(self._h, p.data_ptr(), len(prompts[i]), news[i])
                if sid < 0:
                    if not sid_of:
                        _native.rt_check(sid)
                    break
                sid_of[sid] = i
                pending.pop(0)
            progressed = self._step(max_active)
            done = [sid for sid in sid_of if lib.kh_eng_seq_done(self._h, sid)]
            if done:
                for sid, toks in zip(done, self._collect(done)):
                    outs[sid_of.pop(sid)] = toks
            if not progressed and not pending and not sid_of:
                break
            if not progressed and not sid_of and pending:
                raise _native.NativeError("generate: cannot admit the next sequence")
        ms = (self._timer() - t0) * 1e3
        return outs, self._stats(), ms

    def generate_group(self, prompt, G, n_new):
        """G samples from one shared prompt: the prompt is prefilled once, all of its blocks are
        shared by reference, the first token of every sample is drawn from the single prefill
        logits row, and a block is copied only when a sample first writes into it
        (infer_generate_group, src/core/infer.c:315-387)."""
        lib = _native.rt()
        lib.kh_eng_reset(self._h)
        t0 = self._timer()
        p = torch.tensor(prompt, dtype=torch.int32)
        parent = _native.rt_check(lib.kh_eng_add(self._h, p.data_ptr(), len(prompt), 0))
        rc, ntok, nseq, npairs = self._plan(1)
        first = self._run(ntok, nseq, rep=G).clone()
        _native.rt_check(lib.kh_eng_commit(self._h, first.data_ptr(), nseq))
        kids = torch.zeros(G, dtype=torch.int32)
        _native.rt_check(lib.kh_eng_fork(self._h, parent, G, n_new, kids.data_ptr()))
        lib.kh_eng_release(self._h, parent)
        _native.rt_check(lib.kh_eng_push_many(self._h, G, kids.data_ptr(), first.data_ptr()))
        while self._step(G):
            pass
        outs = self._collect(kids.tolist())
        ms = (self._timer() - t0) * 1e3
        return outs, self._stats(), ms

    def generate_groups(self, prompts, G, n_new):
        """``generate_group`` for several prompts at once (one GRPO rollout batch): all prompts are
        prefilled in one step, each is forked G ways with its first tokens drawn from its own
        logits row, then all len(prompts) * G samples decode together.  Returns
        ([prompt][g] -> tokens, stats, ms)."""
        lib = _native.rt()
        lib.kh_eng_reset(self._h)
        t0 = self._timer()
        parents = []
        for pr in prompts:
            p = torch.tensor(pr, dtype=torch.int32)
            parents.append(_native.rt_check(lib.kh_eng_add(self._h, p.data_ptr(), len(pr), 0)))
        rc, ntok, nseq, npairs = self._plan(len(prompts))
        assert nseq == len(prompts), "prefill of all prompts must fit one step"
        order = self.h_seq_ids[:nseq].tolist()
        first = self._run(ntok, nseq, rep=G).clone()
        _native.rt_check(lib.kh_eng_commit(self._h, first.data_ptr(), nseq))
        kids_of = {}
        kids = torch.zeros(G, dtype=torch.int32)
        for row, parent in enumerate(order):
            _native.rt_check(lib.kh_eng_fork(self._h, parent, G, n_new, kids.data_ptr()))
            lib.kh_eng_release(self._h, parent)
            kids_of[parent] = kids.tolist()
            _native.rt_check(lib.kh_eng_push_many(self._h, G, kids.data_ptr(), first.data_ptr() + 4 * row * G))
        while self._step(len(prompts) * G):
            pass
        flat = self._collect([k for p in parents for k in kids_of[p]])
        outs = [flat[i * G:(i + 1) * G] for i in range(len(parents))]
        ms = (self._timer() - t0) * 1e3
        return outs, self._stats(), ms

    def kv_bytes_per_position(self):
        return 2 * self.cfg.n_layer * self.Hl * self.hd * self.kc.element_size()


def smoke_decode():
    """Tiny paged decode on cuda:0 (part of the driver's smoke check)."""
    from ..models import Config
    cfg = Config(2, 128, 2, 512, 128, 1)
    m = GPT(cfg, "cuda:0", torch.bfloat16)
    m.init_weights(1234)
    eng = InferEngine(m, block_size=16, max_seqs=5)
    prompt = [(i * 131 + 7) % cfg.vocab for i in range(20)]
    outs, st, ms = eng.generate_group(prompt, 4, 12)
    assert all(len(o) == 32 for o in outs) and all(o == outs[0] for o in outs)
    ops.check_device_status()
    print("smoke: paged decode 4 x 12 tokens, %d blocks peak, %d prefix blocks shared" % (st["blocks_peak"],
                                                                                      st["prefix_blocks_saved"]))
    # a width the persistent decode kernel takes (all layers and the head of a step in one launch)
    cfg = Config(2, 512, 8, 512, 128, 1)
    m = GPT(cfg, "cuda:0", torch.bfloat16)
    m.init_weights(1234)
    eng = InferEngine(m, block_size=16, max_seqs=5)
    outs, st, ms = eng.generate_group(prompt, 4, 12)
    assert eng.persistent and all(len(o) == 32 for o in outs) and all(o == outs[0] for o in outs)
    ops.check_device_status()
    print("smoke: persistent decode kernel, 4 x 12 tokens")
