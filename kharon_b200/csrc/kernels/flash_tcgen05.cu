// Causal FlashAttention forward and backward on tcgen05 tensor cores (sm_100a).
//
// Operates directly on the fused projection buffer qkv [B*T, 3*H*hd] (q | k | v, head-major
// inside each third) and writes merged-head outputs [B*T, H*hd], so the reference's head
// split / merge / unmerge / combine kernels (src/core/kernels.cu:189-228, 468-509) have no
// counterpart here: the strides are folded into the TMA tensor maps.  Replaces
// src/kernels/flash.cu:26-199 (warp-per-row SIMT) and its per-call cudaMalloc (:201-229).
//
// Tiles are [rows x hd] bf16, stored in shared memory as hd/64 slabs of rows x 128 bytes with
// the 128-byte swizzle, exactly as TMA writes them.  The same slab is used as a K-major
// operand (contraction over hd) or as an MN-major operand (contraction over rows) just by
// changing the UMMA descriptor -- e.g. V for O = P V, dO for dV = P^T dO, Q for dK = dS^T Q.
//
// All three kernels are persistent and warp-specialised: a TMA warp streams operand tiles through
// mbarrier-guarded rings, one lane of an MMA warp issues every tcgen05.mma, and the remaining warps
// own the rows of the CTA's tile (softmax in the forward pass, P / dS in the backward pass).  S, dP
// and the accumulators (O; dK and dV; dQ) live in TMEM; finished tiles are staged in shared memory
// and written with TMA stores.  Details stand in front of each kernel.
// backward  delta = rowsum(dO * O); a dK/dV kernel per key tile and a dQ kernel per query tile.
//           No atomics: every output element is produced by exactly one CTA in a fixed order, so
//           gradients are reproducible bit for bit.
//
// All mbarrier waits are bounded (error word code 6); after a timeout the CTA skips its
// stores, releases TMEM and returns.
#include "common.cuh"

#include "flash_short.h"

#define KH_LAUNCH_CHECK(name)                                                     \
  do {                                                                            \
    cudaError_t e_ = cudaGetLastError();                                          \
    if (e_ != cudaSuccess) { kh_set_error(name ": %s", cudaGetErrorString(e_)); return -1; } \
  } while (0)

namespace {

constexpr float LOG2E = 1.4426950408889634f;

struct AttnParams {
  int B, T, H;
  int ld;            // row pitch of qkv / dqkv in elements
  float scale;       // 1/sqrt(hd)
  bf16* out;         // fwd: O [B*T, H*hd];          bwd: unused
  float* lse;        // [B, H, T] natural-log LSE of the scaled scores
  const bf16* o;     // bwd (delta): forward output
  const bf16* dout;  // bwd: dO [B*T, H*hd]
  float* delta;      // [B, H, T]
  bf16* dqkv;        // bwd output
  int* err;
};

// [rows x hd] tile: hd/64 slabs of rows x 128 B
template <int HD>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* m, uint32_t bar, int col0, int row0, int rows) {
#pragma unroll
  for (int s = 0; s < HD / 64; s++) tma_load_2d(dst + s * rows * 128, m, bar, col0 + s * 64, row0);
}
// The items of a persistent CTA, longest first: round r hands them out from the first CTA to the last, the next one from the last to the
// first, so that the longest of a round and the longest of the next do not meet on one CTA: with two or three rounds of causal tiles the
// slowest CTA had 1.7 times the mean (B 2 H 16 T 1777, head width 64: 38 key tiles of 22.7; forward 43.6 us and backward 135, in this order 30.5
// and 97; B 1 H 16 T 4096: 93 and 299, 62 and 200; head width 128 T 1777: 49 and 164, 34 and 131).  In one round, or with equal items, nothing changes.
__device__ __forceinline__ int next_item(int& round, int w) { return 2 * ++round * (int)gridDim.x - 1 - w; }
// UMMA descriptors.  Contraction over the tile's columns (K-major): k-step kk of 16 columns starts
// (kk >> 2) slabs + (kk & 3) * 32 bytes into the tile.  Contraction over the tile's rows (MN-major):
// k-step kk of 16 rows starts kk * 2048 bytes in, slabs are `rows * 128` bytes apart (LBO).
// The MMA warp's single lane issues every product of a CTA, so its instruction count per tcgen05.mma
// bounds the rate: descriptors are built once per tile (dk0 / dmn0) and advanced by compile-time
// constants per k-step (one 64-bit add each).
__device__ __forceinline__ uint64_t dk0(uint32_t base) { return umma_desc_sw128(base, 16, 1024); }
__device__ __forceinline__ uint64_t dmn0(uint32_t base, int rows) { return umma_desc_sw128(base, rows * 128, 1024); }
#define DK(d0, rows, kk) ((d0) + (uint64_t)((((kk) >> 2) * (rows) * 128 + ((kk) & 3) * 32) >> 4))
#define DMN(d0, kk) ((d0) + (uint64_t)(((kk) * 2048) >> 4))
// address of the 16-byte chunk (row, chunk c of 8 bf16) in a K-major tile with `rows` rows
__device__ __forceinline__ uint32_t chunk_addr(uint32_t base, int rows, int row, int c) {
  return base + (c >> 3) * rows * 128 + row * 128 + (((c & 7) ^ (row & 7)) << 4);
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// ================================================================================ forward, warp-specialised
// Persistent CTAs of six warps, two CTAs per SM.  A work item is (batch, head, 128 consecutive
// queries), one thread of warps 0-3 per query row.  Warp 4 streams the Q tile and a two-stage ring of
// (K, V) tiles of 64 keys with TMA; one lane of warp 5 issues every tcgen05.mma.  Per key tile j:
//
//   S(j) = Q K_j^T  -> TMEM (two S buffers)        MMA warp, as soon as K_j has landed
//   softmax warps:     read S(j), online softmax, P(j) -> shared memory (bf16)
//   O   += P(j) V_j   accumulated in TMEM           MMA warp, when P(j) is ready
//
// S(j+1) is already in TMEM when the softmax of tile j ends, and the second CTA of the SM keeps the
// tensor cores and the exponential unit busy while this one waits, loads or stores.  O stays in TMEM
// for the whole item; when a row's running maximum grows by more than 2^8 the row is rescaled in
// place (tcgen05.ld / st), otherwise the older maximum stays the reference of the exponentials,
// which keeps the result exact (the normaliser uses the same reference) and makes rescaling rare
// after the first tiles.  Items are handed out longest first (most key tiles).
template <int HD>
struct FwdWs {
  static constexpr int BQ = 128, BKV = 64, NS = 2;
  static constexpr int Q_BYTES = BQ * HD * 2, KV_BYTES = BKV * HD * 2, P_BYTES = BQ * BKV * 2;
  static constexpr int DATA = Q_BYTES + NS * 2 * KV_BYTES + P_BYTES;
  static constexpr int SMEM = DATA + 256;      // the tiles start at the (1024-byte aligned) base of dynamic shared memory
  static constexpr int THREADS = 192, TMEM_COLS = 256;     // S: 2 x 64 columns, O: HD columns from 128
};

// NSEG = 1: B sequences of equal length T, one set of tensor maps.  NSEG > 1 (prefill of several prompts in one launch): up to
// NSEG sequences of their own lengths, each with its own maps, whose row extents keep a sequence's loads and stores within
// its rows; `seg.pair` lists (sequence, query tile) by falling number of key tiles, an item is a pair and a head.
constexpr int MAX_SEGS = 16, MAX_PAIRS = 512;
template <int NSEG> struct FwdMaps { CUtensorMap q[NSEG], kv[NSEG], o[NSEG]; };
template <int NSEG> struct FwdSegs { int T[NSEG]; uint16_t pair[MAX_PAIRS]; };      // pair = query tile * MAX_SEGS + sequence
template <> struct FwdSegs<1> {};

template <int HD, int NSEG>
__global__ void __launch_bounds__(192, 2)
flash_fwd_ws_kernel(const __grid_constant__ FwdMaps<NSEG> maps, const __grid_constant__ FwdSegs<NSEG> seg, const AttnParams p,
                    int n_items, int n_qt) {
  using C = FwdWs<HD>;
  constexpr int BQ = C::BQ, BKV = C::BKV, NS = C::NS;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t sQ = base, sKV = sQ + C::Q_BYTES, sP = sKV + NS * 2 * C::KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::DATA);
  const uint32_t b0 = smem_u32(bars);
  // K and V stages are released separately: a K stage as soon as S(j) has retired, a V stage after PV(j)
  const uint32_t bar_qfull = b0, bar_qfree = b0 + 8, bar_kfull = b0 + 16, bar_kfree = bar_kfull + 8 * NS,
                 bar_vfull = bar_kfree + 8 * NS, bar_vfree = bar_vfull + 8 * NS,
                 bar_sfull = bar_vfree + 8 * NS, bar_pready = bar_sfull + 16, bar_odone = bar_pready + 8,
                 bar_ofree = bar_odone + 8, bar_epi = bar_ofree + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 + 4 * NS + 2 + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(bar_qfull, 1); mbar_init(bar_qfree, 1);
    for (int s = 0; s < NS; s++) {
      mbar_init(bar_kfull + 8 * s, 1); mbar_init(bar_kfree + 8 * s, 1);
      mbar_init(bar_vfull + 8 * s, 1); mbar_init(bar_vfree + 8 * s, 1);
    }
    mbar_init(bar_sfull, 1); mbar_init(bar_sfull + 8, 1);
    mbar_init(bar_pready, 4); mbar_init(bar_odone, 1); mbar_init(bar_ofree, 4); mbar_init(bar_epi, 128);
    *abort_flag = (base & 1023u) ? 6 : 0;       // swizzled tiles need the 1024-byte alignment
    if (base & 1023u) atomicCAS(p.err, 0, 6);
    mbar_fence_init();
    tma_prefetch_desc(&maps.q[0]);
    tma_prefetch_desc(&maps.kv[0]);
    tma_prefetch_desc(&maps.o[0]);
  }
  if (warp == 5) { tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();

  const int d = p.H * HD, BH = p.B * p.H;
  // item w -> (query tile, batch, head) and its number of key tiles; the tiles that see the most keys come first.  Returns
  // the index of the item's tensor maps; b is 0 there when every sequence has its own.
  auto decode = [&](int w, int& b, int& h, int& q0, int& n) -> int {
    if constexpr (NSEG > 1) {
      const int pr = seg.pair[w / p.H], sg = pr % MAX_SEGS;
      b = 0; h = w % p.H; q0 = pr / MAX_SEGS * BQ;
      n = (min(q0 + BQ, seg.T[sg]) + BKV - 1) / BKV;
      return sg;
    } else {
      const int qt = n_qt - 1 - w / BH, bh = w % BH;
      b = bh / p.H; h = bh % p.H; q0 = qt * BQ;
      n = (min(q0 + BQ, p.T) + BKV - 1) / BKV;
      return 0;
    }
  };
  const bool live = *abort_flag == 0;

  if (warp == 4) {
    // ------------------------------------------------------------------ TMA producer
    if (live && elect_one()) {
      int ic = 0, kvc = 0;
      bool ok = true;
      for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w), ic++) {
        int b, h, q0, n;
        const int sg = decode(w, b, h, q0, n);
        if (!mbar_wait(bar_qfree, (ic & 1) ^ 1, abort_flag, 6, p.err)) break;
        mbar_expect_tx(bar_qfull, C::Q_BYTES);
        load_tile<HD>(sQ, &maps.q[sg], bar_qfull, h * HD, b * p.T + q0, BQ);
        for (int j = 0; j < n; j++, kvc++) {
          const int s = kvc % NS;
          const uint32_t par = ((kvc / NS) & 1) ^ 1;
          const uint32_t sk = sKV + s * 2 * C::KV_BYTES, sv = sk + C::KV_BYTES;
          if (!mbar_wait(bar_kfree + 8 * s, par, abort_flag, 6, p.err)) { ok = false; break; }
          mbar_expect_tx(bar_kfull + 8 * s, C::KV_BYTES);
          load_tile<HD>(sk, &maps.kv[sg], bar_kfull + 8 * s, d + h * HD, b * p.T + j * BKV, BKV);
          if (!mbar_wait(bar_vfree + 8 * s, par, abort_flag, 6, p.err)) { ok = false; break; }
          mbar_expect_tx(bar_vfull + 8 * s, C::KV_BYTES);
          load_tile<HD>(sv, &maps.kv[sg], bar_vfull + 8 * s, 2 * d + h * HD, b * p.T + j * BKV, BKV);
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer
    if (live && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BKV, 0, 0);
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, HD, 0, 1);
      int ic = 0, pc = 0, kvc = 0;
      bool ok = true;
      const uint64_t dQ0 = dk0(sQ), dP0 = dk0(sP);
      for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w), ic++) {
        int b, h, q0, n;
        decode(w, b, h, q0, n);
        if (!mbar_wait(bar_qfull, ic & 1, abort_flag, 6, p.err)) break;
        const int kv_base = kvc;
        for (int j = 0; j <= n && ok; j++) {
          if (j < n) {
            const int s = kvc % NS;
            if (!mbar_wait(bar_kfull + 8 * s, (kvc / NS) & 1, abort_flag, 6, p.err)) { ok = false; break; }
            kvc++;
            tc_fence_after();
            const uint32_t sk = sKV + s * 2 * C::KV_BYTES;
            const uint32_t tS = tmem + (j & 1) * 64;
            const uint64_t dK0 = dk0(sk);
#pragma unroll
            for (int kk = 0; kk < HD / 16; kk++) umma_f16_ss(tS, DK(dQ0, BQ, kk), DK(dK0, BKV, kk), idesc_s, kk > 0);
            umma_commit(bar_sfull + 8 * (j & 1));
            umma_commit(bar_kfree + 8 * s);
            if (j == n - 1) umma_commit(bar_qfree);         // last use of this item's Q
          }
          if (j >= 1) {
            const int jj = j - 1;
            const int s = (kv_base + jj) % NS;
            const uint32_t sv = sKV + s * 2 * C::KV_BYTES + C::KV_BYTES;
            if (!mbar_wait(bar_vfull + 8 * s, ((kv_base + jj) / NS) & 1, abort_flag, 6, p.err)) { ok = false; break; }
            // the previous item's O has been read out
            if (jj == 0 && !mbar_wait(bar_ofree, (ic & 1) ^ 1, abort_flag, 6, p.err)) { ok = false; break; }
            if (!mbar_wait(bar_pready, pc & 1, abort_flag, 6, p.err)) { ok = false; break; }
            pc++;
            tc_fence_after();
            const uint64_t dV0 = dmn0(sv, BKV);
#pragma unroll
            for (int kk = 0; kk < BKV / 16; kk++)
              umma_f16_ss(tmem + 128, DK(dP0, BQ, kk), DMN(dV0, kk), idesc_o, (jj > 0 || kk > 0));
            umma_commit(bar_odone);
            umma_commit(bar_vfree + 8 * s);
          }
        }
      }
    }
  } else if (live) {
    // ------------------------------------------------------------------ softmax warps
    const int row = tid;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    const uint32_t tO = tmem + 128 + lane_off;
    const float sl2 = p.scale * LOG2E;
    uint32_t sph = 0;                          // parity of each S buffer
    int odc = 0, epc = 0;
    bool ok = true;
    for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w)) {
      int b, h, q0, n;
      const int sg = decode(w, b, h, q0, n);
      const int qpos = q0 + row;
      float m_ref = -INFINITY, l_run = 0.f;     // reference maximum (scaled to log2 units) and normaliser
      for (int j = 0; j < n; j++) {
        const int buf = j & 1;
        if (!mbar_wait(bar_sfull + 8 * buf, (sph >> buf) & 1, abort_flag, 6, p.err)) { ok = false; break; }
        sph ^= 1u << buf;
        tc_fence_after();
        const int k0 = j * BKV;
        bool waited = false;
        uint32_t pk[32];
        if (k0 > qpos - lane + 31) {           // all keys come after the queries of this warp (never the first tile)
#pragma unroll
          for (int i = 0; i < 32; i++) pk[i] = 0u;
        } else {
          uint32_t r[64];
          const uint32_t tS = tmem + buf * 64 + lane_off;
          tmem_ld32(tS, r);
          tmem_ld32(tS + 32, r + 32);
          tmem_ld_wait();
          if (k0 + BKV - 1 > qpos - lane) {      // the diagonal: mask keys after the query
#pragma unroll
            for (int i = 0; i < 64; i++)
              if (k0 + i > qpos) r[i] = 0xff800000u;
          }
          // maximum of the raw scores over four independent chains (the scale is positive)
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            mx[0] = fmaxf(mx[0], __uint_as_float(r[i])); mx[1] = fmaxf(mx[1], __uint_as_float(r[i + 1]));
            mx[2] = fmaxf(mx[2], __uint_as_float(r[i + 2])); mx[3] = fmaxf(mx[3], __uint_as_float(r[i + 3]));
          }
          const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2;
          if (j == 0) {
            m_ref = mt;
          } else {
            const bool grow = mt > m_ref + 8.f;
            if (__any_sync(0xffffffffu, grow)) {
              // rescale O in place: PV(j-1) must have retired, PV(j) is issued only after P(j) below
              if (!mbar_wait(bar_odone, odc & 1, abort_flag, 6, p.err)) { ok = false; break; }
              odc++;
              waited = true;
              tc_fence_after();
              const float alpha = grow ? exp2f(m_ref - mt) : 1.f;
#pragma unroll 1
              for (int c = 0; c < HD; c += 32) {
                uint32_t o[32];
                tmem_ld32(tO + c, o);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                tmem_st32(tO + c, o);
              }
              tmem_st_wait();
              l_run *= alpha;
              if (grow) m_ref = mt;
            }
          }
          f32x2 rs0 = 0, rs1 = 0;
          const f32x2 sl = mk2(sl2, sl2), nm = mk2(-m_ref, -m_ref);
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            const f32x2 e0 = fma2(mk2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), sl, nm);
            const f32x2 e1 = fma2(mk2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), sl, nm);
            const f32x2 p0 = mk2(exp2f(lo2(e0)), exp2f(hi2(e0))), p1 = mk2(exp2f(lo2(e1)), exp2f(hi2(e1)));
            rs0 = add2(rs0, p0); rs1 = add2(rs1, p1);
            pk[i >> 1] = pack2(p0);
            pk[(i >> 1) + 1] = pack2(p1);
          }
          l_run += (lo2(rs0) + hi2(rs0)) + (lo2(rs1) + hi2(rs1));
        }
        if (j >= 1 && !waited) {      // PV(j-1) no longer reads the P buffer
          if (!mbar_wait(bar_odone, odc & 1, abort_flag, 6, p.err)) { ok = false; break; }
          odc++;
        }
#pragma unroll
        for (int c = 0; c < 8; c++)
          st_shared_v4(chunk_addr(sP, BQ, row, c), pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_pready);
      }
      if (!ok) break;
      if (!mbar_wait(bar_odone, odc & 1, abort_flag, 6, p.err)) { ok = false; break; }
      odc++;
      tc_fence_after();
      // O tile -> bf16 -> the P buffer (free now) in the swizzled tile layout, 64 columns at a time -> one
      // TMA store per slab; rows past the end of the sequence are clipped by the tensor map
      const float inv = 1.f / l_run;
#pragma unroll 1
      for (int hf = 0; hf < HD / 64; hf++) {
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t o[32];
          tmem_ld32(tO + hf * 64 + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; q++)
            st_shared_v4(chunk_addr(sP, BQ, row, (c >> 3) + q),
                         pack_bf16(__uint_as_float(o[8 * q]) * inv, __uint_as_float(o[8 * q + 1]) * inv),
                         pack_bf16(__uint_as_float(o[8 * q + 2]) * inv, __uint_as_float(o[8 * q + 3]) * inv),
                         pack_bf16(__uint_as_float(o[8 * q + 4]) * inv, __uint_as_float(o[8 * q + 5]) * inv),
                         pack_bf16(__uint_as_float(o[8 * q + 6]) * inv, __uint_as_float(o[8 * q + 7]) * inv));
        }
        fence_proxy_async_smem();
        mbar_arrive(bar_epi);
        if (!mbar_wait(bar_epi, epc & 1, abort_flag, 6, p.err)) { ok = false; break; }
        epc++;
        if (tid == 0) {
          tma_store_3d(&maps.o[sg], sP, h * HD + hf * 64, q0, b);
          bulk_commit();
          bulk_wait_read_all();           // the buffer may be overwritten (next slab, next item's P)
        }
        mbar_arrive(bar_epi);
        if (!mbar_wait(bar_epi, epc & 1, abort_flag, 6, p.err)) { ok = false; break; }
        epc++;
      }
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ofree);
      if (qpos < p.T && p.lse) p.lse[((size_t)b * p.H + h) * p.T + qpos] = (m_ref + log2f(l_run)) / LOG2E;
    }
    if (tid == 0) bulk_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

// ================================================================================ delta
// delta[b,h,t] = sum_e dO[b,t,h,e] * O[b,t,h,e].  One warp per row of O / dO: the lanes read the row in
// 16-byte pieces (512 contiguous bytes per step), a head is HD / 8 adjacent lanes, summed with shuffles.
template <int HD>
__global__ void flash_delta_kernel(const bf16* __restrict__ o, const bf16* __restrict__ dout, float* __restrict__ delta,
                                   int B, int T, int H) {
  pdl_wait();
  pdl_launch_dependents();
  const long row = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= (long)B * T) return;
  constexpr int LPH = HD / 8;                      // lanes per head
  const int d = H * HD;
  const uint4* a = reinterpret_cast<const uint4*>(o + row * d);
  const uint4* g = reinterpret_cast<const uint4*>(dout + row * d);
  const int b = (int)(row / T), t = (int)(row % T);
  for (int c0 = 0; c0 < d / 8; c0 += 32) {
    const int c = c0 + lane;
    float s = 0.f;
    if (c < d / 8) {
      const uint4 x = __ldg(a + c), y = __ldg(g + c);
      const float2 x0 = unpack_bf16(x.x), x1 = unpack_bf16(x.y), x2 = unpack_bf16(x.z), x3 = unpack_bf16(x.w);
      const float2 y0 = unpack_bf16(y.x), y1 = unpack_bf16(y.y), y2 = unpack_bf16(y.z), y3 = unpack_bf16(y.w);
      s = (x0.x * y0.x + x0.y * y0.y) + (x1.x * y1.x + x1.y * y1.y) + (x2.x * y2.x + x2.y * y2.y) + (x3.x * y3.x + x3.y * y3.y);
    }
#pragma unroll
    for (int off = LPH / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (c < d / 8 && (lane % LPH) == 0) delta[((size_t)b * H + c / LPH) * T + t] = s;
  }
}

// ================================================================================ backward, warp-specialised
// Both backward kernels are persistent with ten warps: eight compute warps (two
// threads per row of the CTA's 128-row tile, each taking 32 of a sub-tile's 64 columns), a TMA warp
// and an MMA warp.  The other sequence dimension is walked in sub-tiles of 64 through a four-stage
// TMA ring, so S and dP take 64 TMEM columns each and fit twice: the MMA warp issues S(t+1),
// dP(t+1) while the compute warps turn S(t), dP(t) into P(t), dS(t), and issues the accumulating
// products of sub-tile t as soon as those are in shared memory.  Gradients stay in TMEM for the
// whole item.  Work items are handed out longest first.
// TWO (head width 64): S, dP and the gradients take half of the tensor memory when S and dP are held once, and two ring stages
// half of the shared memory, so two CTAs share an SM and fill each other's gaps in the chain S -> tcgen05.ld -> exponentials ->
// shared memory -> accumulating products.  B32 H8 T256: dK/dV 26.8 -> 21.5 us, dQ 20.6 -> 16.7.
// Head width 128, or no more items than SMs (B32 H4 T128: 7.6 us with one CTA, 8.3 with this form): one CTA with two S / dP buffers.
template <int HD, bool TWO>
struct BwdWs {
  static constexpr int BT = 128, BS = 64, NS = TWO ? 2 : 4, CTAS = TWO ? 2 : 1;
  static constexpr int BUFS = TWO ? 1 : 2, ACC = 2 * BUFS * 64;            // S / dP buffers; first TMEM column of the gradients
  static constexpr int CW = TWO ? 16 : 32;                                 // columns a compute thread takes from TMEM at a time
  static constexpr int TILE = BT * HD * 2, SUB = BS * HD * 2, PS_BYTES = BT * BS * 2;
  static constexpr int THREADS = 320, TMEM_COLS = TWO ? 256 : 512;
  // dK/dV: K, V tiles; ring of (Q, dO) sub-tiles; P^T and dS^T; lse / delta of two sub-tiles
  static constexpr int DATA_KV = 2 * TILE + NS * 2 * SUB + 2 * PS_BYTES + 2 * 128 * 4;
  static constexpr int SMEM_KV = DATA_KV + 256;
  // dQ: Q, dO tiles; ring of (K, V) sub-tiles; dS, with 16 KB behind it so that the pair stages the dQ tile
  static constexpr int DATA_Q = 2 * TILE + NS * 2 * SUB + 2 * PS_BYTES;
  static constexpr int SMEM_Q = DATA_Q + 256;
};

// One arrival per warp: the writes of its lanes are ordered before it by the warp barrier (an arrival per thread is 32 updates
// of the barrier word one after the other).
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
template <int W> __device__ __forceinline__ void tmem_cols(uint32_t a, uint32_t* r) {
  if (W == 32) tmem_ld32(a, r); else tmem_ld16(a, r);
}

// ---- dK, dV: item = (batch, head, 128 keys); sub-tiles of 64 queries from the diagonal to the end
// ONE_TILE (head width 128, up to 128 positions, one key tile per item, more than four items per SM): the MMA role is entered by
// lane 0.  With the elected lane the kernel is faster on longer sequences and few items (whole backward B 32 H8 T1777: 1357 -> 1130 us;
// T 66, 32 items: 16.4 -> 15.8) and slower there (T 100, 4800 items: 386 -> 419).
template <int HD, bool TWO, bool ONE_TILE>
__global__ void __launch_bounds__(320, BwdWs<HD, TWO>::CTAS)
flash_dkv_ws_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_q,
                    const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_dqkv, const AttnParams p,
                    int n_items, int n_kt) {
  using C = BwdWs<HD, TWO>;
  constexpr int BT = C::BT, BS = C::BS, NS = C::NS, BUFS = C::BUFS, ACC = C::ACC, CW = C::CW;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t sK = base, sV = sK + C::TILE, sQD = sV + C::TILE, sP = sQD + NS * 2 * C::SUB, sDS = sP + C::PS_BYTES;
  float* s_stat = reinterpret_cast<float*>(smem_raw + 2 * C::TILE + NS * 2 * C::SUB + 2 * C::PS_BYTES);   // [2][128]: lse | delta
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::DATA_KV);
  const uint32_t b0 = smem_u32(bars);
  const uint32_t bar_kvfull = b0, bar_kvfree = b0 + 8, bar_qfull = b0 + 16, bar_qfree = bar_qfull + 8 * NS,
                 bar_sfull = bar_qfree + 8 * NS, bar_ready = bar_sfull + 16, bar_gdone = bar_ready + 8,
                 bar_accfree = bar_gdone + 8, bar_stat = bar_accfree + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 + 2 * NS + 2 + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(bar_kvfull, 1); mbar_init(bar_kvfree, 1);
    for (int s = 0; s < NS; s++) { mbar_init(bar_qfull + 8 * s, 1); mbar_init(bar_qfree + 8 * s, 1); }
    mbar_init(bar_sfull, 1); mbar_init(bar_sfull + 8, 1);
    mbar_init(bar_ready, 8); mbar_init(bar_gdone, 1); mbar_init(bar_accfree, 8); mbar_init(bar_stat, 8);
    *abort_flag = (base & 1023u) ? 6 : 0;
    if (base & 1023u) atomicCAS(p.err, 0, 6);
    mbar_fence_init();
    tma_prefetch_desc(&map_kv); tma_prefetch_desc(&map_q); tma_prefetch_desc(&map_do); tma_prefetch_desc(&map_dqkv);
  }
  if (warp == 9) { tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();
  const int d = p.H * HD, BH = p.B * p.H;
  // key tile 0 sees every query: longest items first
  auto decode = [&](int w, int& b, int& h, int& k0, int& n) {
    const int jt = w / BH, bh = w % BH;
    b = bh / p.H; h = bh % p.H; k0 = jt * BT;
    n = (p.T - k0 + BS - 1) / BS;
  };
  const bool live = *abort_flag == 0;

  if (warp == 8) {
    if (live && elect_one()) {
      int ic = 0, qc = 0;
      bool ok = true;
      for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w), ic++) {
        int b, h, k0, n;
        decode(w, b, h, k0, n);
        if (!mbar_wait(bar_kvfree, (ic & 1) ^ 1, abort_flag, 6, p.err)) break;
        mbar_expect_tx(bar_kvfull, 2 * C::TILE);
        load_tile<HD>(sK, &map_kv, bar_kvfull, d + h * HD, b * p.T + k0, BT);
        load_tile<HD>(sV, &map_kv, bar_kvfull, 2 * d + h * HD, b * p.T + k0, BT);
        for (int t = 0; t < n; t++, qc++) {
          const int s = qc % NS;
          if (!mbar_wait(bar_qfree + 8 * s, ((qc / NS) & 1) ^ 1, abort_flag, 6, p.err)) { ok = false; break; }
          const uint32_t sq = sQD + s * 2 * C::SUB, sdo = sq + C::SUB;
          mbar_expect_tx(bar_qfull + 8 * s, 2 * C::SUB);
          load_tile<HD>(sq, &map_q, bar_qfull + 8 * s, h * HD, b * p.T + k0 + t * BS, BS);
          load_tile<HD>(sdo, &map_do, bar_qfull + 8 * s, h * HD, b * p.T + k0 + t * BS, BS);
        }
      }
    }
  } else if (warp == 9) {
    if (live && (ONE_TILE ? lane == 0 : elect_one())) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BS, 0, 0);
      constexpr uint32_t idesc_g = umma_idesc_bf16(128, HD, 0, 1);
      int ic = 0, qc = 0, rc = 0;
      bool ok = true;
      const uint64_t dK0 = dk0(sK), dV0 = dk0(sV), dP0 = dk0(sP), dDS0 = dk0(sDS);
      for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w), ic++) {
        int b, h, k0, n;
        decode(w, b, h, k0, n);
        if (!mbar_wait(bar_kvfull, ic & 1, abort_flag, 6, p.err)) break;
        const int q_base = qc;
        for (int t = 0; t <= n && ok; t++) {
          // with one S / dP buffer the next products may overwrite it once P and dS of the sub-tile before are in shared memory
          if (BUFS == 1 && t >= 1) {
            if (!mbar_wait(bar_ready, rc & 1, abort_flag, 6, p.err)) { ok = false; break; }
            rc++;
            tc_fence_after();
          }
          if (t < n) {
            const int s = qc % NS;
            if (!mbar_wait(bar_qfull + 8 * s, (qc / NS) & 1, abort_flag, 6, p.err)) { ok = false; break; }
            qc++;
            tc_fence_after();
            const uint32_t sq = sQD + s * 2 * C::SUB, sdo = sq + C::SUB;
            const uint32_t tS = tmem + (t & (BUFS - 1)) * 64, tDP = tmem + BUFS * 64 + (t & (BUFS - 1)) * 64;
            const uint64_t dq0 = dk0(sq), ddo0 = dk0(sdo);
#pragma unroll
            for (int kk = 0; kk < HD / 16; kk++) {
              umma_f16_ss(tS, DK(dK0, BT, kk), DK(dq0, BS, kk), idesc_s, kk > 0);
              umma_f16_ss(tDP, DK(dV0, BT, kk), DK(ddo0, BS, kk), idesc_s, kk > 0);
            }
            umma_commit(bar_sfull + 8 * (t & (BUFS - 1)));
            if (t == n - 1) umma_commit(bar_kvfree);        // K and V are only read by these products
          }
          if (t >= 1) {
            const int tt = t - 1, s = (q_base + tt) % NS;
            const uint32_t sq = sQD + s * 2 * C::SUB, sdo = sq + C::SUB;
            if (tt == 0 && !mbar_wait(bar_accfree, (ic & 1) ^ 1, abort_flag, 6, p.err)) { ok = false; break; }
            if (BUFS == 2) {
              if (!mbar_wait(bar_ready, rc & 1, abort_flag, 6, p.err)) { ok = false; break; }
              rc++;
            }
            tc_fence_after();
            const uint64_t mdo0 = dmn0(sdo, BS), mq0 = dmn0(sq, BS);
#pragma unroll
            for (int kk = 0; kk < BS / 16; kk++) {
              umma_f16_ss(tmem + ACC, DK(dP0, BT, kk), DMN(mdo0, kk), idesc_g, (tt > 0 || kk > 0));
              umma_f16_ss(tmem + ACC + HD, DK(dDS0, BT, kk), DMN(mq0, kk), idesc_g, (tt > 0 || kk > 0));
            }
            umma_commit(bar_gdone);
            umma_commit(bar_qfree + 8 * s);
          }
        }
      }
    }
  } else if (live) {
    const int row = tid & 127, half = tid >> 7;          // this thread: key row `row`, columns [32 half, 32 half + 32) of a sub-tile
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const float sl2 = p.scale * LOG2E;
    uint32_t sph = 0;                          // parity of each S buffer
    int uses = 0, obs = 0, stc = 0;
    bool ok = true;
    for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w)) {
      int b, h, k0, n;
      decode(w, b, h, k0, n);
      const int kpos = k0 + row;
      const size_t stat0 = ((size_t)b * p.H + h) * p.T;
      // threads 0-63 fetch the lse of query tid of sub-tile t, threads 64-127 its delta.  The value is only
      // touched (scaled, stored) at the end of the iteration, so the load is in flight during the sub-tile.
      // They are kept negated: -lse in log2 units (-inf past the end, so that P is 0 there), -delta.
      const float stat_mul = tid < 64 ? -LOG2E : -1.f;
      auto fetch_stat = [&](int t) -> float {
        const int qp = k0 + t * BS + (tid & 63);
        if (tid >= 128 || t >= n || qp >= p.T) return tid < 64 ? INFINITY : 0.f;
        return __ldg((tid < 64 ? p.lse : p.delta) + stat0 + qp);
      };
      if (tid < 128) s_stat[tid] = fetch_stat(0) * stat_mul;
      warp_arrive(bar_stat, lane);
      if (!mbar_wait(bar_stat, stc & 1, abort_flag, 6, p.err)) break;
      stc++;
      for (int t = 0; t < n; t++) {
        const int sb = t & 1, buf = t & (BUFS - 1);
        const float next_stat = fetch_stat(t + 1);
        const float* st = s_stat + sb * 128;
        if (!mbar_wait(bar_sfull + 8 * buf, (sph >> buf) & 1, abort_flag, 6, p.err)) { ok = false; break; }
        sph ^= 1u << buf;
        tc_fence_after();
        const int q0s = k0 + t * BS;
        const int c = half * 32;
        // what this warp sees of the sub-tile: 32 keys and 32 queries, all before the keys, across the diagonal or all after
        const int ahead = kpos - lane - (q0s + c);
        const bool none = ahead > 31, diag = ahead > -31;
        const f32x2 sl = mk2(sl2, sl2), sc = mk2(p.scale, p.scale);
        uint32_t pp[16], ds[16];
        if (none) {
#pragma unroll
          for (int e = 0; e < 16; e++) pp[e] = ds[e] = 0u;
        } else {
#pragma unroll
          for (int w = 0; w < 32; w += CW) {
            uint32_t rs[CW], rd[CW];
            tmem_cols<CW>(tmem + buf * 64 + lane_off + c + w, rs);
            tmem_cols<CW>(tmem + BUFS * 64 + buf * 64 + lane_off + c + w, rd);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < CW; e += 4) {
              const int q0 = c + w + e;
              const ulonglong2 nl = *reinterpret_cast<const ulonglong2*>(st + q0), nd = *reinterpret_cast<const ulonglong2*>(st + 64 + q0);
#pragma unroll
              for (int u = 0; u < 4; u += 2) {
                const f32x2 x = fma2(mk2(__uint_as_float(rs[e + u]), __uint_as_float(rs[e + u + 1])), sl, u ? nl.y : nl.x);
                const f32x2 pr = mk2(exp2f(lo2(x)), exp2f(hi2(x)));
                const f32x2 dp = add2(mk2(__uint_as_float(rd[e + u]), __uint_as_float(rd[e + u + 1])), u ? nd.y : nd.x);
                pp[(w + e + u) >> 1] = pack2(pr);
                ds[(w + e + u) >> 1] = pack2(mul2(mul2(pr, dp), sc));
              }
            }
            if (diag) {                        // 0 whatever the statistics of a query that comes before the key (NaN, -inf)
#pragma unroll
              for (int e = 0; e < CW; e += 2) {
                const int q = q0s + c + w + e;
                const uint32_t keep = (kpos > q ? 0u : 0xffffu) | (kpos > q + 1 ? 0u : 0xffff0000u);
                pp[(w + e) >> 1] &= keep;
                ds[(w + e) >> 1] &= keep;
              }
            }
          }
        }
        // the products that read P^T / dS^T of the previous sub-tile have retired
        while (obs < uses) {
          if (!mbar_wait(bar_gdone, obs & 1, abort_flag, 6, p.err)) { ok = false; break; }
          obs++;
        }
        if (!ok) break;
#pragma unroll
        for (int g = 0; g < 4; g++) {
          st_shared_v4(chunk_addr(sP, BT, row, (c >> 3) + g), pp[4 * g], pp[4 * g + 1], pp[4 * g + 2], pp[4 * g + 3]);
          st_shared_v4(chunk_addr(sDS, BT, row, (c >> 3) + g), ds[4 * g], ds[4 * g + 1], ds[4 * g + 2], ds[4 * g + 3]);
        }
        uses++;
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_ready);
        if (tid < 128) s_stat[(sb ^ 1) * 128 + tid] = next_stat * stat_mul;
        warp_arrive(bar_stat, lane);
        if (!mbar_wait(bar_stat, stc & 1, abort_flag, 6, p.err)) { ok = false; break; }
        stc++;
      }
      if (!ok) break;
      while (obs < uses) {      // the last accumulating products have retired
        if (!mbar_wait(bar_gdone, obs & 1, abort_flag, 6, p.err)) { ok = false; break; }
        obs++;
      }
      if (!ok) break;
      tc_fence_after();
      // dV, then dK: TMEM -> bf16 -> the P^T / dS^T buffers (free now, 2 x 16 KB = one 128 x 128 tile in the
      // swizzled layout) -> one TMA store per 64-column slab; rows past the end of the sequence are clipped
#pragma unroll 1
      for (int which = 0; which < 2; which++) {
        const uint32_t tacc = tmem + ACC + which * HD + lane_off;
#pragma unroll 1
        for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 32) {
          uint32_t r1[32];
          tmem_ld32(tacc + c, r1);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 4; g++)
            st_shared_v4(chunk_addr(sP, BT, row, (c >> 3) + g),
                         pack_bf16(__uint_as_float(r1[8 * g]), __uint_as_float(r1[8 * g + 1])),
                         pack_bf16(__uint_as_float(r1[8 * g + 2]), __uint_as_float(r1[8 * g + 3])),
                         pack_bf16(__uint_as_float(r1[8 * g + 4]), __uint_as_float(r1[8 * g + 5])),
                         pack_bf16(__uint_as_float(r1[8 * g + 6]), __uint_as_float(r1[8 * g + 7])));
        }
        fence_proxy_async_smem();
        warp_arrive(bar_stat, lane);
        if (!mbar_wait(bar_stat, stc & 1, abort_flag, 6, p.err)) { ok = false; break; }
        stc++;
        if (tid == 0) {
          const int col0 = (which == 0 ? 2 * d : d) + h * HD;
#pragma unroll
          for (int sl = 0; sl < HD / 64; sl++) tma_store_3d(&map_dqkv, sP + sl * C::PS_BYTES, col0 + sl * 64, k0, b);
          bulk_commit();
          bulk_wait_read_all();
        }
        warp_arrive(bar_stat, lane);
        if (!mbar_wait(bar_stat, stc & 1, abort_flag, 6, p.err)) { ok = false; break; }
        stc++;
      }
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_accfree);
    }
    if (tid == 0) bulk_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

// ---- dQ: item = (batch, head, 128 queries); sub-tiles of 64 keys up to the diagonal
template <int HD, bool TWO>
__global__ void __launch_bounds__(320, BwdWs<HD, TWO>::CTAS)
flash_dq_ws_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                   const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_dqkv, const AttnParams p,
                   int n_items, int n_qt) {
  using C = BwdWs<HD, TWO>;
  constexpr int BT = C::BT, BS = C::BS, NS = C::NS, BUFS = C::BUFS, ACC = C::ACC, CW = C::CW;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t sQ = base, sDO = sQ + C::TILE, sKV = sDO + C::TILE, sDS = sKV + NS * 2 * C::SUB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::DATA_Q);
  const uint32_t b0 = smem_u32(bars);
  const uint32_t bar_qfull = b0, bar_qfree = b0 + 8, bar_kvfull = b0 + 16, bar_kvfree = bar_kvfull + 8 * NS,
                 bar_sfull = bar_kvfree + 8 * NS, bar_ready = bar_sfull + 16, bar_gdone = bar_ready + 8, bar_accfree = bar_gdone + 8,
                 bar_epi = bar_accfree + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 + 2 * NS + 2 + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(bar_qfull, 1); mbar_init(bar_qfree, 1);
    for (int s = 0; s < NS; s++) { mbar_init(bar_kvfull + 8 * s, 1); mbar_init(bar_kvfree + 8 * s, 1); }
    mbar_init(bar_sfull, 1); mbar_init(bar_sfull + 8, 1);
    mbar_init(bar_ready, 8); mbar_init(bar_gdone, 1); mbar_init(bar_accfree, 8); mbar_init(bar_epi, 8);
    *abort_flag = (base & 1023u) ? 6 : 0;
    if (base & 1023u) atomicCAS(p.err, 0, 6);
    mbar_fence_init();
    tma_prefetch_desc(&map_kv); tma_prefetch_desc(&map_q); tma_prefetch_desc(&map_do); tma_prefetch_desc(&map_dqkv);
  }
  if (warp == 9) { tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();
  const int d = p.H * HD, BH = p.B * p.H;
  // the last query tile sees the most keys: longest items first
  auto decode = [&](int w, int& b, int& h, int& q0, int& n) {
    const int qt = n_qt - 1 - w / BH, bh = w % BH;
    b = bh / p.H; h = bh % p.H; q0 = qt * BT;
    n = (min(q0 + BT, p.T) + BS - 1) / BS;
  };
  const bool live = *abort_flag == 0;

  if (warp == 8) {
    if (live && elect_one()) {
      int ic = 0, kvc = 0;
      bool ok = true;
      for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w), ic++) {
        int b, h, q0, n;
        decode(w, b, h, q0, n);
        if (!mbar_wait(bar_qfree, (ic & 1) ^ 1, abort_flag, 6, p.err)) break;
        mbar_expect_tx(bar_qfull, 2 * C::TILE);
        load_tile<HD>(sQ, &map_q, bar_qfull, h * HD, b * p.T + q0, BT);
        load_tile<HD>(sDO, &map_do, bar_qfull, h * HD, b * p.T + q0, BT);
        for (int j = 0; j < n; j++, kvc++) {
          const int s = kvc % NS;
          if (!mbar_wait(bar_kvfree + 8 * s, ((kvc / NS) & 1) ^ 1, abort_flag, 6, p.err)) { ok = false; break; }
          const uint32_t sk = sKV + s * 2 * C::SUB, sv = sk + C::SUB;
          mbar_expect_tx(bar_kvfull + 8 * s, 2 * C::SUB);
          load_tile<HD>(sk, &map_kv, bar_kvfull + 8 * s, d + h * HD, b * p.T + j * BS, BS);
          load_tile<HD>(sv, &map_kv, bar_kvfull + 8 * s, 2 * d + h * HD, b * p.T + j * BS, BS);
        }
      }
    }
  } else if (warp == 9) {
    if (live && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BS, 0, 0);
      constexpr uint32_t idesc_g = umma_idesc_bf16(128, HD, 0, 1);
      int ic = 0, kvc = 0, rc = 0;
      bool ok = true;
      const uint64_t dQ0 = dk0(sQ), dDO0 = dk0(sDO), dDS0 = dk0(sDS);
      for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w), ic++) {
        int b, h, q0, n;
        decode(w, b, h, q0, n);
        if (!mbar_wait(bar_qfull, ic & 1, abort_flag, 6, p.err)) break;
        const int kv_base = kvc;
        for (int j = 0; j <= n && ok; j++) {
          if (BUFS == 1 && j >= 1) {              // see the dK / dV kernel
            if (!mbar_wait(bar_ready, rc & 1, abort_flag, 6, p.err)) { ok = false; break; }
            rc++;
            tc_fence_after();
          }
          if (j < n) {
            const int s = kvc % NS;
            if (!mbar_wait(bar_kvfull + 8 * s, (kvc / NS) & 1, abort_flag, 6, p.err)) { ok = false; break; }
            kvc++;
            tc_fence_after();
            const uint32_t sk = sKV + s * 2 * C::SUB, sv = sk + C::SUB;
            const uint32_t tS = tmem + (j & (BUFS - 1)) * 64, tDP = tmem + BUFS * 64 + (j & (BUFS - 1)) * 64;
            const uint64_t dk_0 = dk0(sk), dv_0 = dk0(sv);
#pragma unroll
            for (int kk = 0; kk < HD / 16; kk++) {
              umma_f16_ss(tS, DK(dQ0, BT, kk), DK(dk_0, BS, kk), idesc_s, kk > 0);
              umma_f16_ss(tDP, DK(dDO0, BT, kk), DK(dv_0, BS, kk), idesc_s, kk > 0);
            }
            umma_commit(bar_sfull + 8 * (j & (BUFS - 1)));
            if (j == n - 1) umma_commit(bar_qfree);         // Q and dO are only read by these products
          }
          if (j >= 1) {
            const int jj = j - 1, s = (kv_base + jj) % NS;
            const uint32_t sk = sKV + s * 2 * C::SUB;
            if (jj == 0 && !mbar_wait(bar_accfree, (ic & 1) ^ 1, abort_flag, 6, p.err)) { ok = false; break; }
            if (BUFS == 2) {
              if (!mbar_wait(bar_ready, rc & 1, abort_flag, 6, p.err)) { ok = false; break; }
              rc++;
            }
            tc_fence_after();
            const uint64_t mk0 = dmn0(sk, BS);
#pragma unroll
            for (int kk = 0; kk < BS / 16; kk++)
              umma_f16_ss(tmem + ACC, DK(dDS0, BT, kk), DMN(mk0, kk), idesc_g, (jj > 0 || kk > 0));
            umma_commit(bar_gdone);
            umma_commit(bar_kvfree + 8 * s);
          }
        }
      }
    }
  } else if (live) {
    const int row = tid & 127, half = tid >> 7;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const float sl2 = p.scale * LOG2E;
    uint32_t sph = 0;                          // parity of each S buffer
    int uses = 0, obs = 0, epc = 0;
    bool ok = true;
    for (int round = 0, w = blockIdx.x; ok && w < n_items; w = next_item(round, w)) {
      int b, h, q0, n;
      decode(w, b, h, q0, n);
      const int qpos = q0 + row;
      const bool qvalid = qpos < p.T;
      const size_t sidx = ((size_t)b * p.H + h) * p.T + qpos;
      const float my_lse = qvalid ? p.lse[sidx] * LOG2E : INFINITY;
      const float my_delta = qvalid ? p.delta[sidx] : 0.f;
      for (int j = 0; j < n; j++) {
        const int buf = j & (BUFS - 1);
        if (!mbar_wait(bar_sfull + 8 * buf, (sph >> buf) & 1, abort_flag, 6, p.err)) { ok = false; break; }
        sph ^= 1u << buf;
        tc_fence_after();
        const int k0 = j * BS;
        const int c = half * 32;
        const int ahead = k0 + c - (qpos - lane);        // as in the dK / dV kernel
        const bool none = ahead > 31, diag = ahead > -31;
        const f32x2 sl = mk2(sl2, sl2), sc = mk2(p.scale, p.scale), nl = mk2(-my_lse, -my_lse), nd = mk2(-my_delta, -my_delta);
        uint32_t ds[16];
        if (none) {
#pragma unroll
          for (int e = 0; e < 16; e++) ds[e] = 0u;
        } else {
#pragma unroll
          for (int w = 0; w < 32; w += CW) {
            uint32_t rs[CW], rd[CW];
            tmem_cols<CW>(tmem + buf * 64 + lane_off + c + w, rs);
            tmem_cols<CW>(tmem + BUFS * 64 + buf * 64 + lane_off + c + w, rd);
            tmem_ld_wait();
            if (diag) {
#pragma unroll
              for (int e = 0; e < CW; e++)
                if (k0 + c + w + e > qpos) rs[e] = 0xff800000u;         // -inf: dS is 0
            }
#pragma unroll
            for (int e = 0; e < CW; e += 2) {
              const f32x2 x = fma2(mk2(__uint_as_float(rs[e]), __uint_as_float(rs[e + 1])), sl, nl);
              const f32x2 pr = mk2(exp2f(lo2(x)), exp2f(hi2(x)));
              ds[(w + e) >> 1] = pack2(mul2(mul2(pr, add2(mk2(__uint_as_float(rd[e]), __uint_as_float(rd[e + 1])), nd)), sc));
            }
          }
        }
        while (obs < uses) {
          if (!mbar_wait(bar_gdone, obs & 1, abort_flag, 6, p.err)) { ok = false; break; }
          obs++;
        }
        if (!ok) break;
#pragma unroll
        for (int g = 0; g < 4; g++)
          st_shared_v4(chunk_addr(sDS, BT, row, (c >> 3) + g), ds[4 * g], ds[4 * g + 1], ds[4 * g + 2], ds[4 * g + 3]);
        uses++;
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_ready);
      }
      if (!ok) break;
      while (obs < uses) {
        if (!mbar_wait(bar_gdone, obs & 1, abort_flag, 6, p.err)) { ok = false; break; }
        obs++;
      }
      if (!ok) break;
      tc_fence_after();
      // dQ: TMEM -> bf16 -> staging tile (the dS buffer and the 16 KB behind it) -> one TMA store per slab
#pragma unroll 1
      for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 32) {
        uint32_t r1[32];
        tmem_ld32(tmem + ACC + lane_off + c, r1);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; g++)
          st_shared_v4(chunk_addr(sDS, BT, row, (c >> 3) + g),
                       pack_bf16(__uint_as_float(r1[8 * g]), __uint_as_float(r1[8 * g + 1])),
                       pack_bf16(__uint_as_float(r1[8 * g + 2]), __uint_as_float(r1[8 * g + 3])),
                       pack_bf16(__uint_as_float(r1[8 * g + 4]), __uint_as_float(r1[8 * g + 5])),
                       pack_bf16(__uint_as_float(r1[8 * g + 6]), __uint_as_float(r1[8 * g + 7])));
      }
      fence_proxy_async_smem();
      warp_arrive(bar_epi, lane);
      if (!mbar_wait(bar_epi, epc & 1, abort_flag, 6, p.err)) { ok = false; break; }
      epc++;
      if (tid == 0) {
#pragma unroll
        for (int sl = 0; sl < HD / 64; sl++) tma_store_3d(&map_dqkv, sDS + sl * C::PS_BYTES, h * HD + sl * 64, q0, b);
        bulk_commit();
        bulk_wait_read_all();
      }
      warp_arrive(bar_epi, lane);
      if (!mbar_wait(bar_epi, epc & 1, abort_flag, 6, p.err)) { ok = false; break; }
      epc++;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_accfree);
    }
    if (tid == 0) bulk_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

template <typename K>
int set_smem(K kernel, int bytes, const char* name) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) { kh_set_error("%s: cannot opt in to %d bytes of shared memory: %s", name, bytes, cudaGetErrorString(e)); return -1; }
  return 0;
}

static int num_sms_attn() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 148;
}

template <int HD, int NSEG>
int launch_fwd_items(const FwdMaps<NSEG>& maps, const FwdSegs<NSEG>& seg, const AttnParams& p, int n_items, int n_qt, cudaStream_t st) {
  using C = FwdWs<HD>;
  static bool once = false;
  if (!once) { if (set_smem(flash_fwd_ws_kernel<HD, NSEG>, C::SMEM, "flash_fwd")) return -1; once = true; }
  const int ctas = 2 * num_sms_attn();                  // two CTAs per SM
  KH_LAUNCH((flash_fwd_ws_kernel<HD, NSEG>), n_items < ctas ? n_items : ctas, C::THREADS, C::SMEM, st, maps, seg, p, n_items, n_qt);
  KH_LAUNCH_CHECK("flash_fwd");
  return 0;
}
template <int NSEG>
int fwd_maps(FwdMaps<NSEG>& maps, int i, const void* qkv, void* out, int B, int T, int H, int hd, int ld) {
  const size_t rows = (size_t)B * T;
  const CUtensorMap* mq = kh_tmap_2d_bf16(qkv, rows, 3 * H * hd, ld, 128, 64);
  const CUtensorMap* mkv = kh_tmap_2d_bf16(qkv, rows, 3 * H * hd, ld, 64, 64);
  const CUtensorMap* mo = kh_tmap_3d_bf16(out, (uint64_t)H * hd, T, B, (uint64_t)H * hd, (uint64_t)T * H * hd, 128, 64);
  if (!mq || !mkv || !mo) return -1;
  maps.q[i] = *mq; maps.kv[i] = *mkv; maps.o[i] = *mo;
  return 0;
}
template <int HD>
int launch_fwd(const void* qkv, const AttnParams& p, cudaStream_t st) {
  FwdMaps<1> maps;
  if (fwd_maps(maps, 0, qkv, p.out, p.B, p.T, p.H, HD, p.ld)) return -1;
  const int n_qt = (p.T + 127) / 128;
  return launch_fwd_items<HD, 1>(maps, FwdSegs<1>{}, p, p.B * p.H * n_qt, n_qt, st);
}
// Sequences of rows [row0[i], row0[i] + len[i]) of qkv and out, as many per launch as the maps and the list of pairs hold.
template <int HD>
int launch_fwd_varlen(const bf16* qkv, AttnParams p, const int* row0, const int* len, int n_seg, cudaStream_t st) {
  bf16* out = p.out;
  for (int s0 = 0; s0 < n_seg;) {
    FwdMaps<MAX_SEGS> maps;
    FwdSegs<MAX_SEGS> seg;
    int n = 0, pairs = 0, most = 0;
    while (s0 + n < n_seg && n < MAX_SEGS && pairs + (len[s0 + n] + 127) / 128 <= MAX_PAIRS) {
      const int i = s0 + n, q = (len[i] + 127) / 128;
      if (fwd_maps(maps, n, qkv + (size_t)row0[i] * p.ld, out + (size_t)row0[i] * p.H * HD, 1, len[i], p.H, HD, p.ld)) return -1;
      seg.T[n] = len[i];
      pairs += q;
      most = q > most ? q : most;
      n++;
    }
    if (n == 0 || (n == 1 && s0 + 1 == n_seg)) {      // longer than the list, or one alone: by itself, without the sixteen sets of maps
      p.B = 1; p.T = len[s0]; p.out = out + (size_t)row0[s0] * p.H * HD;
      if (launch_fwd<HD>(qkv + (size_t)row0[s0] * p.ld, p, st)) return -1;
      s0++;
      continue;
    }
    for (int i = n; i < MAX_SEGS; i++) { maps.q[i] = maps.q[0]; maps.kv[i] = maps.kv[0]; maps.o[i] = maps.o[0]; seg.T[i] = 0; }
    int at = 0;
    for (int qt = most - 1; qt >= 0; qt--)
      for (int i = 0; i < n; i++)
        if (qt < (seg.T[i] + 127) / 128) seg.pair[at++] = (uint16_t)(qt * MAX_SEGS + i);
    p.B = 1; p.T = 0;
    if (launch_fwd_items<HD, MAX_SEGS>(maps, seg, p, pairs * p.H, most, st)) return -1;
    s0 += n;
  }
  return 0;
}

template <int HD, bool TWO>
int launch_bwd_as(const void* qkv, const AttnParams& p, cudaStream_t st) {
  using C = BwdWs<HD, TWO>;
  const size_t rows = (size_t)p.B * p.T;
  const CUtensorMap* mq = kh_tmap_2d_bf16(qkv, rows, 3 * p.H * HD, p.ld, 128, 64);
  const CUtensorMap* md = kh_tmap_2d_bf16(p.dout, rows, p.H * HD, p.H * HD, 128, 64);
  const CUtensorMap* mq64 = kh_tmap_2d_bf16(qkv, rows, 3 * p.H * HD, p.ld, 64, 64);
  const CUtensorMap* md64 = kh_tmap_2d_bf16(p.dout, rows, p.H * HD, p.H * HD, 64, 64);
  const CUtensorMap* mg = kh_tmap_3d_bf16(p.dqkv, (uint64_t)3 * p.H * HD, p.T, p.B, (uint64_t)p.ld, (uint64_t)p.T * p.ld, 128, 64);
  if (!mq || !md || !mq64 || !md64 || !mg) return -1;
  KH_LAUNCH((flash_delta_kernel<HD>), (unsigned)((rows * 32 + 255) / 256), 256, 0, st, p.o, p.dout, p.delta, p.B, p.T, p.H);
  const int n_t = (p.T + 127) / 128;
  auto dkv = HD == 128 && n_t == 1 && p.B * p.H > 4 * num_sms_attn() ? flash_dkv_ws_kernel<HD, TWO, HD == 128> : flash_dkv_ws_kernel<HD, TWO, false>;
  static bool once = false;
  if (!once) {
    if (set_smem(flash_dkv_ws_kernel<HD, TWO, HD == 128>, C::SMEM_KV, "flash_dkv") ||
        set_smem(flash_dkv_ws_kernel<HD, TWO, false>, C::SMEM_KV, "flash_dkv") || set_smem(flash_dq_ws_kernel<HD, TWO>, C::SMEM_Q, "flash_dq")) return -1;
    once = true;
  }
  const int n_items = p.B * p.H * n_t;
  const int ctas = C::CTAS * num_sms_attn();
  const int grid = n_items < ctas ? n_items : ctas;
  KH_LAUNCH(dkv, grid, C::THREADS, C::SMEM_KV, st, *mq, *mq64, *md64, *mg, p, n_items, n_t);
  KH_LAUNCH((flash_dq_ws_kernel<HD, TWO>), grid, C::THREADS, C::SMEM_Q, st, *mq, *md, *mq64, *mg, p, n_items, n_t);
  KH_LAUNCH_CHECK("flash_bwd");
  return 0;
}
template <int HD>
int launch_bwd(const void* qkv, const AttnParams& p, cudaStream_t st) {
  if (HD == 64 && (long)p.B * p.H * ((p.T + 127) / 128) > num_sms_attn()) return launch_bwd_as<HD, HD == 64>(qkv, p, st);
  return launch_bwd_as<HD, false>(qkv, p, st);
}

// Whether flash_short.cu takes the sequences: up to 64 positions always.  Its cost is the arithmetic of mma.sync on the rows that are there, that of
// the kernels here the latency of an item per resident CTA.  Head width 64: B 32-1000 H8 T 33-64 0.4 to 0.93 of the time forward, 0.3 to 0.91
// backward, before its loads were asynchronous.  Head width 128, us (short / tcgen05): forward T 33, 2080 items 16.1 / 28.3; T 48, 8000 65.0 / 86.6;
// T 64, 960 12.7 / 17.0 and 8000 84.5 / 89.9; backward T 56, 592 items 20.9 / 38.8; T 64, 8000 318 / 475.
static bool use_short(int T) { return T >= 1 && T <= KH_FLASH_SHORT_T; }

}  // namespace

extern "C" int kh_flash_fwd(const void* qkv, void* out, void* lse, int B, int T, int H, int hd, int ld, float scale,
                            void* stream) {
  if (hd != 64 && hd != 128) { kh_set_error("flash: head dim %d is not supported (64 or 128)", hd); return -1; }
  if (use_short(T)) return kh_flash_short_fwd(qkv, out, lse, B, T, H, hd, ld, scale, stream);
  AttnParams p = {};
  p.B = B; p.T = T; p.H = H; p.ld = ld; p.scale = scale; p.out = (bf16*)out; p.lse = (float*)lse;
  p.err = kh_error_word_dev();
  return hd == 64 ? launch_fwd<64>(qkv, p, (cudaStream_t)stream) : launch_fwd<128>(qkv, p, (cudaStream_t)stream);
}

// Causal attention of several sequences of different lengths: sequence i occupies rows [row0[i], row0[i] + len[i]) of qkv
// (pitch ld) and out; row0 and len are host arrays.  No log-sum-exps are written.
extern "C" int kh_flash_fwd_varlen(const void* qkv, void* out, const void* row0, const void* len, int n_seg, int H, int hd, int ld,
                                   float scale, void* stream) {
  if (hd != 64 && hd != 128) { kh_set_error("flash: head dim %d is not supported (64 or 128)", hd); return -1; }
  for (int i = 0; i < n_seg; i++)
    if (((const int*)row0)[i] < 0 || ((const int*)len)[i] < 1) { kh_set_error("flash_varlen: sequence %d is empty", i); return -1; }
  AttnParams p = {};
  p.H = H; p.ld = ld; p.scale = scale; p.out = (bf16*)out;
  p.err = kh_error_word_dev();
  return hd == 64 ? launch_fwd_varlen<64>((const bf16*)qkv, p, (const int*)row0, (const int*)len, n_seg, (cudaStream_t)stream)
                  : launch_fwd_varlen<128>((const bf16*)qkv, p, (const int*)row0, (const int*)len, n_seg, (cudaStream_t)stream);
}

extern "C" int kh_flash_bwd(const void* qkv, const void* out, const void* dout, const void* lse, void* dqkv,
                            void* delta, int B, int T, int H, int hd, int ld, float scale, void* stream) {
  if (hd != 64 && hd != 128) { kh_set_error("flash: head dim %d is not supported (64 or 128)", hd); return -1; }
  if (use_short(T)) return kh_flash_short_bwd(qkv, out, dout, lse, dqkv, delta, B, T, H, hd, ld, scale, stream);
  AttnParams p = {};
  p.B = B; p.T = T; p.H = H; p.ld = ld; p.scale = scale; p.lse = (float*)lse; p.o = (const bf16*)out;
  p.dout = (const bf16*)dout; p.delta = (float*)delta; p.dqkv = (bf16*)dqkv;
  p.err = kh_error_word_dev();
  return hd == 64 ? launch_bwd<64>(qkv, p, (cudaStream_t)stream) : launch_bwd<128>(qkv, p, (cudaStream_t)stream);
}
