// All transformer layers (and the vocabulary head) of one decode step in ONE persistent kernel (sm_100a).
//
// A decode step of G <= 32 sequences is latency-bound: its per-layer chain LayerNorm -> qkv -> paged
// attention -> proj -> LayerNorm -> fc/GELU -> fcproj moves a few megabytes of weights, and as five
// launches per layer (src/core/infer.c:204-262 issues more than twenty) every link of the chain pays
// a launch, a pipeline prologue and a split-K hand-off.  Here one cooperative grid (one CTA per SM)
// walks the chain for all layers.
//
//   phase A  xs = LN1(x)            qkv  = xs Wqkv^T + b                        (N = 3d, K = d)
//   phase B  per (sequence, head): append k, v to the paged cache, att = softmax(q K^T) V
//   phase C                         xmid = att Wproj^T + b + x                  (N = d,  K = d)
//   phase D  xs = LN2(xmid)         act  = gelu(bf16(xs Wfc^T + b))             (N = 4d, K = d)
//   phase E                         x    = act Wfcproj^T + b + xmid             (N = d,  K = 4d)
//   head     xs = LNf(x[rows])      logits = xs Whead^T                         (N = V,  K = d)
//
// Links.  What bounds the step is the trip from the CTAs that write an activation to those that read
// it.  There is no grid barrier: an activation travels as 8-byte packets {two bf16 columns, epoch},
// written with one 64-bit store and polled by its readers until the epoch of this launch and layer
// shows (a 64-bit access is single-copy atomic, so a packet with the right epoch holds the right
// data).  One trip through L2 replaces the release fence, the arrival atomic, the polled counter and
// the fetch of a barrier; a CTA without work in a phase does not take part in it.  Packets double the
// bytes of an activation, which are a few KB per row.  A buffer is overwritten one layer later; by then every
// reader is done, because each phase's output depends on all rows and columns of the one before it.
// Measured, L24 d1024 with the head, context 160, a captured step with embedding and sampler: 468 us for one
// sequence and 520 for eight (grid barriers and weights held in registers: 1000 and 1090; the weights alone
// take 106 us at the copy bandwidth).
//
// Linear phases.  A work unit is 16 output columns (8 in phases C and E, whose N is only d); S warps share
// a unit, each multiplying its K / S slice, and a CTA of 16 (8) warps works on 16 / S (8 / S) units at a time.  S is
// the smallest split whose slice fits a sub-step, and larger where that spreads a narrow product over more
// CTAs in the same number of turns.  Every lane copies the eight (sixteen) 16-byte pieces of weights that it will use
// into its own slots of shared memory with cp.async (no registers are held and no thread waits for another's
// copy); the first turn's weights of a phase are requested before its activations are polled, the next turn's
// are requested under the products of this one (a second set of slots for up to eight rows, else as a slot has been read), and the units of later phases are prefetched
// into L2 in bulk.  The products are mma.sync m16n8k16 with the weights as the 16-row operand and eight sequences
// as the columns: tcgen05's 128-row tiles, TMEM round trip and operand staging are the latency this kernel
// exists to avoid (the large-M GEMMs of training and prefill use them).  The K order inside a 32-wide block
// is permuted identically for both operands so that every lane fetches 16 contiguous bytes.  Phases behind a
// LayerNorm read the normalised rows from shared memory (pitch padded by 64 bytes, conflict-free); the others read their operand fragments straight from the packets.  Partial sums of the S
// warps meet in shared memory and are added in warp order.
//
// Attention.  W warps share a (sequence, head) item; a key is read by HD / 8 lanes in 16-byte pieces and
// the running softmax is kept per lane group and merged once.  The first four (eight) keys and values of
// every group are requested before the queries are polled (cached positions do not depend on this step).
//
// Every wait is bounded: status code 9 in the library error word, an abort word for the other CTAs.
// Numerics follow the five-kernel path: bf16 activations between phases, fp32 accumulation, LayerNorm
// statistics in two passes, GELU applied to the bf16-rounded pre-activation.
#include "common.cuh"

namespace {

constexpr int MAX_WARPS = 16;
constexpr int PAD = 32;                       // bf16 elements of padding per activation row (64 bytes)
constexpr int MAX_ROWS = 32;
constexpr int ATT_PITCH = 128 + 4;            // floats per warp of the attention hand-off: 128 outputs, maximum, sum
constexpr int SMEM_LIMIT = 227 * 1024;

// Warps of a CTA (2^LGW) and what follows: 16-byte weight slots per lane (one sub-step; 64 KB a CTA) and the bytes between them.
// Eight warps for up to eight rows, where index arithmetic that every warp repeats weighs most (L24 d1024 G = 1 / 8: 489 / 538 us
// against 507 / 565 with sixteen; d2048 G = 4: 1179 against 1248), sixteen beyond, where rows and keys are spread over more
// warps (G = 16 / 32: 764 / 1217 against 781 / 1320).
template <int LGW> struct Cfg {
  static constexpr int WARPS = 1 << LGW, THREADS = 32 * WARPS, NLD = 128 / WARPS;
  static constexpr uint32_t SLOT = THREADS * 16;
  static constexpr bool DB = LGW == 3;        // two sets of slots: shared memory has room for them up to eight rows
};
#define CFG using C_ = Cfg<LGW>; constexpr int WARPS = C_::WARPS, THREADS = C_::THREADS, NLD = C_::NLD; constexpr uint32_t SLOT = C_::SLOT; (void)WARPS; (void)THREADS; (void)NLD; (void)SLOT

constexpr uint32_t WBUF = 65536;              // bytes of a set of weight slots

// Thread index, read anew in every phase: index arithmetic derived from it would otherwise be kept in registers (and
// spilled) across the whole layer loop.
__device__ __forceinline__ int tid_fresh() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

struct LayerW {               // bf16 pointers of one layer (device array, one entry per layer)
  const bf16 *ln1_w, *ln1_b, *qkv_w, *qkv_b, *proj_w, *proj_b, *ln2_w, *ln2_b, *fc_w, *fc_b, *fcproj_w, *fcproj_b;
};

struct DecodeParams {
  int G, d, H, hd, L, bs, max_lb, max_ctx;
  int lgs_a, lgs_c, lgs_d, lgs_e, lgs_h, lgw;    // log2 of the warps per unit of each product and per attention item
  const LayerW* layers;
  bf16* x;                                // [G, d] in: embedded tokens, out: last layer's output
  uint64_t *xp, *midp, *qkvp, *attp, *actp;   // packets: [32, d/2], [32, d/2], [32, 3d/2], [32, d/2], [32, 4d/2]
  bf16 *kc, *vc;                          // [L, blocks, bs, H, hd]
  size_t layer_elems;
  const int *pos, *slot, *btab;
  // optional head: logits[g, :V] = LNf(x[rows[g]]) Whead^T
  const bf16 *head_w, *lnf_w, *lnf_b;
  bf16* logits;
  int ld_logits, V, n_rows;
  const int* rows;
  uint32_t* ctl;                          // [0] epochs used by earlier launches, [1] abort, [2] CTAs that left
  float scale;
  uint64_t wait_ns;
  int* err;
  uint32_t bs_mul;                        // ceil(2^32 / bs); 0 when one block holds every position
  // j / bs by multiplication: exact for j < max_ctx, since max_ctx * bs stays below 2^32
  __device__ __forceinline__ int block_of(int j) const { return bs == 1 ? j : (int)__umulhi((uint32_t)j, bs_mul); }
};

struct Shared {               // small control block behind the data regions
  LayerW lw[4];               // records of this layer and the next two
  int item_pos[MAX_WARPS], item_slot[MAX_WARPS];    // position and slot of each warp's first attention item (constant over the layers)
  int item_row[MAX_WARPS][8][8];                // cache rows of its first keys, per lane group
  volatile int abort_flag;
};

__device__ __forceinline__ uint4 ldg_stream(const void* p) {      // read-once data: do not keep it in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_older() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }     // all but the last group
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void l2_prefetch_bulk(const void* p, uint32_t bytes) {       // 16-byte aligned, multiple of 16
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ---- packets
__device__ __forceinline__ void ld_packets(uint64_t& a, uint64_t& b, const uint64_t* p) {     // two packets, 16-byte aligned
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ uint64_t ld_packet(const uint64_t* p) {
  uint64_t a;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return a;
}
__device__ __forceinline__ void st_packet(uint64_t* p, uint32_t data, uint32_t epoch) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((uint64_t)epoch << 32) | data) : "memory");
}
// After an unsuccessful poll: true when the wait is over (limit reached, or another thread or CTA gave up).  Inline on
// purpose: a call would make the compiler keep the values in flight in local memory.
__device__ __forceinline__ bool poll_expired(uint32_t& it, uint64_t& t0, Shared* sh, const DecodeParams& p) {
  if ((++it & 127) != 0) return false;
  if (sh->abort_flag) return true;
  uint32_t a;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(p.ctl + 1) : "memory");
  const uint64_t now = kh_globaltimer();
  if (t0 == 0) t0 = now;
  if (a == 0 && now - t0 <= p.wait_ns) return false;
  if (a == 0) {
    atomicCAS(p.err, 0, 9);
    atomicExch(p.ctl + 1, 1u);
  }
  sh->abort_flag = 1;
  return true;
}
// Reads N pairs of packets (pair i from addr(i), when use(i)) once all of them carry `epoch`; out[i] = four columns.
template <int N, class Use, class Addr>
__device__ __forceinline__ void read_pairs(uint2 (&out)[N], Use use, Addr addr, uint32_t epoch, const DecodeParams& p, Shared* sh) {
  uint32_t it = 0;
  uint64_t t0 = 0;
#pragma unroll 1
  while (true) {
    uint64_t a[N], b[N];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; i++) {
      a[i] = b[i] = (uint64_t)epoch << 32;
      if (use(i)) ld_packets(a[i], b[i], addr(i));
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
      ok = ok && (uint32_t)(a[i] >> 32) == epoch && (uint32_t)(b[i] >> 32) == epoch;
      out[i] = make_uint2((uint32_t)a[i], (uint32_t)b[i]);
    }
    if (ok || poll_expired(it, t0, sh, p)) return;
  }
}
__device__ __forceinline__ uint32_t read_one(const uint64_t* q, uint32_t epoch, const DecodeParams& p, Shared* sh) {
  uint32_t it = 0;
  uint64_t t0 = 0;
#pragma unroll 1
  while (true) {
    const uint64_t a = ld_packet(q);
    if ((uint32_t)(a >> 32) == epoch || poll_expired(it, t0, sh, p)) return (uint32_t)a;
  }
}

// One of the five products.
enum Phase { PA, PC, PD, PE, PH };
struct Lin {
  const bf16 *W, *bias;     // [N, K] row-major, [N] (null for the head)
  int N, K, lgs;
  int kind;                 // PA ... PH
  const uint64_t* src;      // packets [32, K / 2] of the input, of epoch e_src (null: plain rows of p.x)
  const uint64_t* res;      // C, E: packets [32, N / 2] of the residual, of epoch e_res (null: plain rows of p.x)
  uint64_t* dst;            // packets [32, N / 2] of the output, epoch e_dst (null for the head)
  uint32_t e_src, e_res, e_dst;
};
// Row groups of eight columns per unit: two fill the 16 rows of an mma (A, D, head); C and E take one (the other half of the
// operand is zero) so that twice as many CTAs have a unit.
// Copies this lane's 16-byte pieces of weight rows 8 (RG u + i) + lane / 4 from column k0 on: slot RG * j + i holds row group
// i of the j-th 32-column step.  Steps below `n` are copied; rows that do not exist are left alone.
template <int LGW, int RG>
__device__ __forceinline__ void copy_w(uint32_t slots, int lane, const Lin& L, int u, int k0, int j, int n) {
  CFG;
  if (j >= n) return;
#pragma unroll
  for (int i = 0; i < RG; i++) {
    const int r = (u * RG + i) * 8 + (lane >> 2);
    if (r < L.N) cp_async16(slots + (j * RG + i) * SLOT, L.W + (size_t)r * L.K + k0 + (lane & 3) * 8 + j * 32);
  }
}
template <int LGW, int RG>
__device__ __forceinline__ void copy_first(uint32_t wbuf, const Lin& L) {
  CFG;
  constexpr int KS = NLD / RG;
  const int tid = tid_fresh(), warp = tid >> 5, U = WARPS >> L.lgs, kw = L.K >> L.lgs;
#pragma unroll
  for (int j = 0; j < KS; j++)
    copy_w<LGW, RG>(wbuf + tid * 16, tid & 31, L, (int)blockIdx.x * U + (warp >> L.lgs), (warp & ((1 << L.lgs) - 1)) * kw, j, kw >> 5);
  cp_async_commit();
}
// ask L2 for the weights of this CTA's units (the first `turns` turns of them); one thread of the last warp, which has the
// least to do at the start of a phase
template <int LGW>
__device__ __forceinline__ void prefetch_units(const bf16* W, int N, int K, int cols, int turns) {
  CFG;
  if (tid_fresh() != THREADS - 32) return;
#pragma unroll 1
  for (int r = 0; r < turns; r++) {
    const int c0 = (r * (int)gridDim.x + (int)blockIdx.x) * cols;
    if (c0 >= N) return;
    l2_prefetch_bulk(W + (size_t)c0 * K, (uint32_t)min(cols, N - c0) * (uint32_t)K * 2u);
  }
}
// LayerNorm gain and bias of a later phase -> shared memory (complete at that phase's first barrier)
template <int LGW>
__device__ __forceinline__ void fetch_ln(bf16* sln, const bf16* w, const bf16* b, int d) {
  CFG;
#pragma unroll 1
  for (int c = tid_fresh(); c < d / 8; c += THREADS) {
    cp_async16(smem_u32(sln + c * 8), w + c * 8);
    cp_async16(smem_u32(sln + d + c * 8), b + c * 8);
  }
  cp_async_commit();
}

// LayerNorm of rows [0, n) into xs, a warp per row: the row is polled, kept in shared memory as it arrived, and
// normalised in place (every lane touches only the 16-byte pieces that it wrote).
template <int LGW>
__device__ __forceinline__ void stage_ln(bf16* xs, const bf16* sln, const Lin& L, int n, const DecodeParams& p, Shared* sh) {
  CFG;
  const int tid = tid_fresh(), warp = tid >> 5, lane = tid & 31;
  const int d = L.K, nch = d / 8;
#pragma unroll 1
  for (int r = warp; r < n; r += WARPS) {
    const int sr = L.kind == PH ? p.rows[r] : r;
    uint4* row = reinterpret_cast<uint4*>(xs + (size_t)r * (d + PAD));
    float sum = 0.f;
#pragma unroll 1
    for (int c0 = lane; c0 < nch; c0 += 128) {
      uint4 v[4];
      if (L.src) {
        const uint64_t* q = L.src + (size_t)sr * (d / 2) + c0 * 4;
        uint2 t[8];
        read_pairs<8>(t, [&](int i) { return c0 + (i >> 1) * 32 < nch; }, [&](int i) { return q + (i >> 1) * 128 + (i & 1) * 2; },
                      L.e_src, p, sh);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = make_uint4(t[2 * i].x, t[2 * i].y, t[2 * i + 1].x, t[2 * i + 1].y);
      } else {
        const uint4* q = reinterpret_cast<const uint4*>(p.x + (size_t)sr * d) + c0;
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = c0 + i * 32 < nch ? __ldcg(q + i * 32) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (c0 + i * 32 >= nch) break;
        row[c0 + i * 32] = v[i];
        const float2 a = unpack_bf16(v[i].x), b = unpack_bf16(v[i].y), cc = unpack_bf16(v[i].z), e = unpack_bf16(v[i].w);
        sum += (a.x + a.y) + (b.x + b.y) + (cc.x + cc.y) + (e.x + e.y);
      }
    }
    const float mean = warp_sum(sum) / (float)d;
    float sq = 0.f;
#pragma unroll 1
    for (int c0 = lane; c0 < nch; c0 += 128)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (c0 + i * 32 >= nch) break;
        const uint4 v = row[c0 + i * 32];
        const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), cc = unpack_bf16(v.z), e = unpack_bf16(v.w);
        const float d0 = a.x - mean, d1 = a.y - mean, d2 = b.x - mean, d3 = b.y - mean, d4 = cc.x - mean, d5 = cc.y - mean,
                    d6 = e.x - mean, d7 = e.y - mean;
        sq += d0 * d0 + d1 * d1 + d2 * d2 + d3 * d3 + d4 * d4 + d5 * d5 + d6 * d6 + d7 * d7;
      }
    const float rstd = rsqrtf(warp_sum(sq) / (float)d + 1e-5f);
    auto n2 = [&](uint32_t x2, uint32_t w2, uint32_t b2) {
      const float2 xv = unpack_bf16(x2), wv = unpack_bf16(w2), bv = unpack_bf16(b2);
      return pack_bf16((xv.x - mean) * rstd * wv.x + bv.x, (xv.y - mean) * rstd * wv.y + bv.y);
    };
#pragma unroll 1
    for (int c0 = lane; c0 < nch; c0 += 64)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int c = c0 + i * 32;
        if (c >= nch) break;
        const uint4 v = row[c], gw = reinterpret_cast<const uint4*>(sln)[c], gb = reinterpret_cast<const uint4*>(sln + d)[c];
        row[c] = make_uint4(n2(v.x, gw.x, gb.x), n2(v.y, gw.y, gb.y), n2(v.z, gw.z, gb.z), n2(v.w, gw.w, gb.w));
      }
  }
}

// One linear phase over rows [0, n) (n <= 8 MT).  The slots hold this warp's weights of its first unit and sub-step
// (copy_first).  LN (A, D, head): the rows go through LayerNorm and shared memory; otherwise (C, E) operand fragments come
// straight from the packets.  One copy of each form serves all layers, which keeps the code small.
template <int LGW, int MT, bool LN>
__device__ __forceinline__ void linear_phase(const DecodeParams& p, const Lin& L, int n, bool last, bf16* xs, const bf16* sln, float* red,
                                             int& flip, Shared* sh, uint32_t wbuf) {
  CFG;
  constexpr bool RES = !LN;
  constexpr int GP = 8 * MT, LGP = MT == 1 ? 3 : (MT == 2 ? 4 : 5);
  constexpr int RG = LN ? 2 : 1, KS = NLD / RG, CU = 8 * RG, LCP = RG == 2 ? 3 : 2;      // steps per sub-step, columns and log2 column pairs per unit
  constexpr int NCH = MT == 1 ? 4 : (MT == 2 ? 2 : 1);          // independent accumulator chains
  const int tid = tid_fresh(), warp = tid >> 5, lane = tid & 31;
  const uint32_t slots = wbuf + tid * 16;
  const int N = L.N, K = L.K, lgs = L.lgs;
  const int S = 1 << lgs, U = WARPS >> lgs, kw = K >> lgs, steps = kw >> 5;
  const int n_units = (N + CU - 1) / CU, stride = (int)gridDim.x * U;
  const int ul = warp >> lgs, ks = warp & (S - 1);
  int unit0 = (int)blockIdx.x * U;
  if (LN) { cp_async_wait_older(); __syncthreads(); }            // gain, bias and layer records are there (the weights need not be); xs is free
  if (unit0 >= n_units) return;                                   // uniform over the CTA
  const int n_out = U * GP * (CU / 2);                            // (unit, row, column pair)
  auto operands = [&](int o, uint32_t& b2, uint64_t& r2) {        // bias and residual packet of output pair o, as they are now
    b2 = 0; r2 = (uint64_t)L.e_res << 32;
    const int g = (o >> LCP) & (GP - 1), col = (unit0 + (o >> (LCP + LGP))) * CU + (o & (CU / 2 - 1)) * 2;
    if (o >= n_out || g >= n || col >= N) return;
    if (L.bias) b2 = __ldg(reinterpret_cast<const unsigned int*>(L.bias + col));
    if (RES) {
      if (!L.res) r2 |= __ldcg(reinterpret_cast<const unsigned int*>(p.x + (size_t)g * N + col));
      else r2 = ld_packet(L.res + ((size_t)g * N + col) / 2);
    }
  };
  bool staged = false;
  constexpr bool DB = C_::DB;
  int wb = 0;                                                     // set of slots that holds the current weights
#pragma unroll 1
  for (; unit0 < n_units; unit0 += stride) {
    const int u = unit0 + ul;
    uint32_t bias2;
    uint64_t res2;
    operands(tid, bias2, res2);
    if (LN && !staged) {
      stage_ln<LGW>(xs, sln, L, n, p, sh);
      __syncthreads();
      staged = true;
    }
    float acc[NCH][MT][4];
#pragma unroll
    for (int c = 0; c < NCH; c++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[c][m][i] = 0.f;
#pragma unroll 1
    for (int s0 = 0; s0 < steps; s0 += KS) {
      const int k0 = ks * kw + s0 * 32, ns = min(KS, steps - s0);
      // the weights that follow these in the same slots: next sub-step, or first sub-step of the next turn
      const bool more = s0 + KS < steps, turn = !more && unit0 + stride < n_units;
      const int nu = more ? u : u + stride, nk = more ? k0 + KS * 32 : ks * kw;
      const int nn = more ? min(KS, steps - s0 - KS) : (turn ? min(KS, steps) : 0);
      // DB: they go into the other set of slots at once, under these products; else into these slots, one by one as they are read
      const uint32_t cur = slots + (DB && wb ? WBUF : 0), nxt = DB ? slots + (wb ? 0 : WBUF) : cur;
      wb ^= 1;
      if (DB && nn > 0) {
#pragma unroll
        for (int j = 0; j < KS; j++) copy_w<LGW, RG>(nxt, lane, L, nu, nk, j, nn);
        cp_async_commit();
      }
      auto wait_weights = [&]() {
        if (DB && nn > 0) cp_async_wait_older(); else cp_async_wait_all();
      };
      if (LN) {
        wait_weights();
        const bf16* xa = xs + (size_t)(lane >> 2) * (K + PAD) + k0 + (lane & 3) * 8;
#pragma unroll
        for (int j = 0; j < KS; j++) {
          if (j < ns) {
            const uint4 w0 = lds128(cur + (2 * j) * SLOT), w1 = lds128(cur + (2 * j + 1) * SLOT);
#pragma unroll
            for (int m = 0; m < MT; m++) {
              const uint4 a = *reinterpret_cast<const uint4*>(xa + (size_t)(m * 8) * (K + PAD) + j * 32);
              mma_bf16(acc[(2 * j) % NCH][m], w0.x, w1.x, w0.y, w1.y, a.x, a.y);
              mma_bf16(acc[(2 * j + 1) % NCH][m], w0.z, w1.z, w0.w, w1.w, a.z, a.w);
            }
          }
          if (!DB) copy_w<LGW, RG>(nxt, lane, L, nu, nk, j, nn);
        }
      } else {
        constexpr int JB = 4 / MT;                                // eight packet pairs in flight per lane
        const uint64_t* q = L.src + (size_t)(lane >> 2) * (K / 2) + (k0 + (lane & 3) * 8) / 2;
#pragma unroll
        for (int j0 = 0; j0 < KS; j0 += JB) {
          if (j0 < ns) {
            uint2 t[8];
            read_pairs<8>(t, [&](int i) { return (i >> 1) % MT * 8 + (lane >> 2) < n && j0 + (i >> 1) / MT < ns; },
                          [&](int i) { return q + (size_t)((i >> 1) % MT * 8) * (K / 2) + (j0 + (i >> 1) / MT) * 16 + (i & 1) * 2; },
                          L.e_src, p, sh);
            if (j0 == 0) wait_weights();
            __syncwarp();
#pragma unroll
            for (int jj = 0; jj < JB; jj++) {
              const int j = j0 + jj;
              if (j < ns) {
                const uint4 w0 = lds128(cur + j * SLOT);
#pragma unroll
                for (int m = 0; m < MT; m++) {
                  const int i = jj * MT + m;
                  mma_bf16(acc[(2 * j) % NCH][m], w0.x, 0u, w0.y, 0u, t[2 * i].x, t[2 * i].y);
                  mma_bf16(acc[(2 * j + 1) % NCH][m], w0.z, 0u, w0.w, 0u, t[2 * i + 1].x, t[2 * i + 1].y);
                }
              }
            }
          }
#pragma unroll
          for (int j = j0; j < j0 + JB; j++)
            if (!DB) copy_w<LGW, RG>(nxt, lane, L, nu, nk, j, nn);
        }
      }
    }
    // partial sums -> shared memory; thread (unit, row, column pair) adds the S slices in order
    float* rb = red + (MT == 4 ? 0 : flip * (WARPS * GP * 16));
    flip ^= 1;
    if (MT == 4) __syncthreads();             // one buffer only: everybody has read the previous turn's
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int i = 0; i < 2 * RG; i++) {
        float v = acc[0][m][i];
#pragma unroll
        for (int c = 1; c < NCH; c++) v += acc[c][m][i];
        rb[((size_t)warp * GP + m * 8 + (lane & 3) * 2 + (i & 1)) * CU + (i >> 1) * 8 + (lane >> 2)] = v;
      }
    __syncthreads();
#pragma unroll 1
    for (int o = tid; o < n_out; o += THREADS) {
      const int g = (o >> LCP) & (GP - 1), cp = (o & (CU / 2 - 1)) * 2, uu = o >> (LCP + LGP), col = (unit0 + uu) * CU + cp;
      if (g >= n || col >= N) continue;
      if (o != tid) operands(o, bias2, res2);
      if (RES && (uint32_t)(res2 >> 32) != L.e_res) res2 = read_one(L.res + ((size_t)g * N + col) / 2, L.e_res, p, sh);
      const float* t = rb + ((size_t)(uu << lgs) * GP + g) * CU + cp;
      float v0 = 0.f, v1 = 0.f;
#pragma unroll 4
      for (int s = 0; s < S; s++) {
        const float2 f = *reinterpret_cast<const float2*>(t + (size_t)s * (GP * CU));
        v0 += f.x; v1 += f.y;
      }
      const float2 b = unpack_bf16(bias2), rr = unpack_bf16((uint32_t)res2);
      v0 += b.x; v1 += b.y;
      if (RES) { v0 += rr.x; v1 += rr.y; }
      if (LN && L.kind == PD) {
        v0 = gelu_tanh(__bfloat162float(__float2bfloat16(v0)));
        v1 = gelu_tanh(__bfloat162float(__float2bfloat16(v1)));
      }
      const uint32_t pk = pack_bf16(v0, v1);
      if (!LN || L.kind != PH) st_packet(L.dst + ((size_t)g * N + col) / 2, pk, L.e_dst);
      if (!LN && last) *reinterpret_cast<uint32_t*>(p.x + (size_t)g * N + col) = pk;
      if (LN && L.kind == PH) {
        bf16* q = p.logits + (size_t)g * p.ld_logits + col;
        if (col + 1 < N && ((uintptr_t)q & 3) == 0) *reinterpret_cast<uint32_t*>(q) = pk;
        else {
          q[0] = __float2bfloat16(v0);
          if (col + 1 < N) q[1] = __float2bfloat16(v1);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Positions a lane group holds at a time: eight for heads of 64 where registers allow it; four for narrow heads, whose eight groups a warp
// cover short contexts in one turn anyway (d256: 59 us a step against 64), and for heads of 128 (no difference).
template <int LGW, int HD> constexpr int keys_ahead() { return LGW == 3 && HD == 64 ? 8 : 4; }
// Phase B.  Appends the new k, v (from the qkv packets) to the paged cache and attends over positions 0..pos.
// The W warps of an item hold W * 32 / (HD / 8) lane groups; group i takes keys i, i + ST, i + 2 ST, ...
template <int LGW, int HD>
__device__ __forceinline__ void attention_phase(const DecodeParams& p, int layer, uint32_t epoch, float* satt, Shared* sh) {
  CFG;
  constexpr int LPK = HD / 8, KPW = 32 / LPK;     // lanes per key, keys of a warp at a time
  constexpr int NB = keys_ahead<LGW, HD>();        // positions a group holds at a time
  const int tid = tid_fresh(), warp = tid >> 5, lane = tid & 31;
  const int W = 1 << p.lgw, slots = WARPS >> p.lgw, ST = W * KPW;
  const int kg = (warp & (W - 1)) * KPW + lane / LPK, e0 = (lane % LPK) * 8;
  const int d = p.d, items = p.G * p.H;
  const bf16* kc = p.kc + (size_t)layer * p.layer_elems;
  const bf16* vc = p.vc + (size_t)layer * p.layer_elems;
#pragma unroll 1
  for (int it0 = (int)blockIdx.x * slots; it0 < items; it0 += (int)gridDim.x * slots) {
    const int item = it0 + (warp >> p.lgw);
    const int t = item / p.H, h = item - t * p.H;
    int pos = -1, slot = -1;
    const bool turn0 = it0 == (int)blockIdx.x * slots;
    if (item < items) {
      pos = turn0 ? sh->item_pos[warp] : __ldg(p.pos + t);
      slot = turn0 ? sh->item_slot[warp] : __ldg(p.slot + t);
    }
    const bool valid = pos >= 0 && pos < p.max_ctx && p.block_of(pos) < p.max_lb && slot >= 0;       // uniform over the item's warps
    if (item < items && !valid && lane == 0) atomicCAS(p.err, 0, 8);
    float m = -INFINITY, l = 0.f, o[8];
#pragma unroll
    for (int k = 0; k < 8; k++) o[k] = 0.f;
    if (valid) {
      const int* bt = p.btab + (size_t)slot * p.max_lb;
      auto row_of = [&](int j) {
        const int jb = p.block_of(j);
        return __ldg(bt + jb) * p.bs + (j - jb * p.bs);
      };
      int row[NB];                    // cache rows of the next positions of this group
      uint4 k4[NB], v4[NB];            // refilled with those positions as soon as they are used
      uint2 qkv2[6];
      float q[8];
      const bool owner = pos % ST == kg;
      const int first = (warp & (W - 1)) * KPW;       // uniform over the warp
      // Turn -1 only requests the first NB keys and values and then waits for the query (and the owner of position `pos`
      // for the new key and value); every other turn uses NB positions and requests the next ones in their place.
#pragma unroll 1
      for (int b0 = -NB * ST; b0 < 0 || first + b0 <= pos; b0 += NB * ST) {
        const int j0 = kg + b0, jn = j0 + NB * ST;
        float s[NB];
#pragma unroll
        for (int i = 0; i < NB; i++)
          if (jn + i * ST < pos) row[i] = b0 < 0 && turn0 ? sh->item_row[warp][lane / LPK][i] : row_of(jn + i * ST);
        if (b0 >= 0) {
#pragma unroll
          for (int i = 0; i < NB; i++) {
            const int j = j0 + i * ST;
            if (j == pos) { k4[i] = make_uint4(qkv2[2].x, qkv2[2].y, qkv2[3].x, qkv2[3].y); v4[i] = make_uint4(qkv2[4].x, qkv2[4].y, qkv2[5].x, qkv2[5].y); }
            if (j > pos) k4[i] = v4[i] = make_uint4(0, 0, 0, 0);
            const float2 a = unpack_bf16(k4[i].x), b = unpack_bf16(k4[i].y), c = unpack_bf16(k4[i].z), e = unpack_bf16(k4[i].w);
            s[i] = a.x * q[0] + a.y * q[1] + b.x * q[2] + b.y * q[3] + c.x * q[4] + c.y * q[5] + e.x * q[6] + e.y * q[7];
          }
        }
        // cached positions only; the same lines of the next layer are requested into L2
#pragma unroll
        for (int i = 0; i < NB; i++)
          if (jn + i * ST < pos) {
            const bf16* c = kc + (size_t)row[i] * d + h * HD + e0;
            k4[i] = ldg_stream(c);
            if (e0 % 64 == 0 && layer + 1 < p.L) prefetch_l2(c + p.layer_elems);
          }
        if (b0 >= 0) {
#pragma unroll
          for (int x = LPK / 2; x > 0; x >>= 1)
#pragma unroll
            for (int i = 0; i < NB; i++) s[i] += __shfl_xor_sync(0xffffffffu, s[i], x);
#pragma unroll
          for (int i = 0; i < NB; i++)
            if (j0 + i * ST > pos) s[i] = -INFINITY;
          float mn = m;
#pragma unroll
          for (int i = 0; i < NB; i++) mn = fmaxf(mn, s[i]);
          const float ref = mn == -INFINITY ? 0.f : mn;
          const float sc = __expf(m - ref);
          m = mn;
          l *= sc;
#pragma unroll
          for (int k = 0; k < 8; k++) o[k] *= sc;
#pragma unroll
          for (int i = 0; i < NB; i++) {
            const float pr = __expf(s[i] - ref);
            l += pr;
            const float2 a = unpack_bf16(v4[i].x), b = unpack_bf16(v4[i].y), c = unpack_bf16(v4[i].z), e = unpack_bf16(v4[i].w);
            o[0] += pr * a.x; o[1] += pr * a.y; o[2] += pr * b.x; o[3] += pr * b.y;
            o[4] += pr * c.x; o[5] += pr * c.y; o[6] += pr * e.x; o[7] += pr * e.y;
          }
        }
#pragma unroll
        for (int i = 0; i < NB; i++)
          if (jn + i * ST < pos) {
            const bf16* c = vc + (size_t)row[i] * d + h * HD + e0;
            v4[i] = ldg_stream(c);
            if (e0 % 64 == 0 && layer + 1 < p.L) prefetch_l2(c + p.layer_elems);
          }
        if (b0 < 0) {
          const uint64_t* qp = p.qkvp + ((size_t)t * 3 * d + h * HD + e0) / 2;
          read_pairs<6>(qkv2, [&](int i) { return i < 2 || owner; }, [&](int i) { return qp + (size_t)(i >> 1) * (d / 2) + (i & 1) * 2; },
                        epoch, p, sh);
          __syncwarp();
          const float2 a = unpack_bf16(qkv2[0].x), b = unpack_bf16(qkv2[0].y), c = unpack_bf16(qkv2[1].x), e = unpack_bf16(qkv2[1].y);
          q[0] = a.x * p.scale; q[1] = a.y * p.scale; q[2] = b.x * p.scale; q[3] = b.y * p.scale;
          q[4] = c.x * p.scale; q[5] = c.y * p.scale; q[6] = e.x * p.scale; q[7] = e.y * p.scale;
        }
      }
      if (owner) {
        const size_t at = (size_t)layer * p.layer_elems + (size_t)row_of(pos) * d + h * HD + e0;
        *reinterpret_cast<uint4*>(p.kc + at) = make_uint4(qkv2[2].x, qkv2[2].y, qkv2[3].x, qkv2[3].y);
        *reinterpret_cast<uint4*>(p.vc + at) = make_uint4(qkv2[4].x, qkv2[4].y, qkv2[5].x, qkv2[5].y);
      }
      // merge the lane groups of the warp
#pragma unroll 1
      for (int x = LPK; x < 32; x <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, x), l2 = __shfl_xor_sync(0xffffffffu, l, x);
        const float mn = fmaxf(m, m2), ref = mn == -INFINITY ? 0.f : mn;
        const float c1 = __expf(m - ref), c2 = __expf(m2 - ref);
        m = mn;
        l = l * c1 + l2 * c2;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const float o2 = __shfl_xor_sync(0xffffffffu, o[k], x);
          o[k] = o[k] * c1 + o2 * c2;
        }
      }
    } else { m = 0.f; l = 1.f; }       // an item with a bad index writes zeros: its row must not stall
    float* mine = satt + warp * ATT_PITCH;
    if (lane < LPK) {
#pragma unroll
      for (int k = 0; k < 8; k += 4) *reinterpret_cast<float4*>(mine + e0 + k) = make_float4(o[k], o[k + 1], o[k + 2], o[k + 3]);
      if (lane == 0) { mine[128] = m; mine[129] = l; }
    }
    __syncthreads();
    // Merge the W warps of each item: lane k (of 16) weighs the k-th partial result of its item.
#pragma unroll 1
    for (int i = tid; i < slots * (HD / 2); i += THREADS) {
      const int sl = i / (HD / 2), e = (i % (HD / 2)) * 2, it = it0 + sl;
      const unsigned mask = HD == 32 ? 0xffffu << (lane & 16) : 0xffffffffu;       // the lanes of this item
      const float* part = satt + (size_t)(sl << p.lgw) * ATT_PITCH;
      const int k16 = lane & 15;
      float c = k16 < W ? part[k16 * ATT_PITCH + 128] : -INFINITY, den = k16 < W ? part[k16 * ATT_PITCH + 129] : 0.f, mx = c;
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(mask, mx, x));
      c = __expf(c - mx);              // (NaN when every score is -inf, as in the kernel chain)
      den *= c;
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) den += __shfl_xor_sync(mask, den, x);
      float v0 = 0.f, v1 = 0.f;
#pragma unroll 4
      for (int k = 0; k < W; k++) {
        const float ck = __shfl_sync(mask, c, (lane & 16) + k);
        const float2 f = *reinterpret_cast<const float2*>(part + k * ATT_PITCH + e);
        v0 += ck * f.x; v1 += ck * f.y;
      }
      const float inv = 1.f / den;
      const int tt = it / p.H;
      if (it < items) st_packet(p.attp + ((size_t)tt * d + (it - tt * p.H) * HD + e) / 2, pack_bf16(v0 * inv, v1 * inv), epoch);
    }
    __syncthreads();               // satt is reused by the next turn or layer
  }
}

template <int MT> constexpr int lg_warps() { return MT == 1 ? 3 : 4; }

template <int MT, int HD>
__global__ void __launch_bounds__(32 << lg_warps<MT>(), 1) decode_layers_k(const __grid_constant__ DecodeParams p) {
  constexpr int LGW = lg_warps<MT>();
  CFG;
  constexpr int GP = 8 * MT;
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t wbuf = smem_u32(smem);
  bf16* xs = reinterpret_cast<bf16*>(smem + (C_::DB ? 2 : 1) * WBUF);
  bf16* sln = xs + (size_t)GP * (p.d + PAD);
  float* red = reinterpret_cast<float*>(sln + 2 * p.d);
  float* satt = red + (MT == 4 ? 1 : 2) * WARPS * GP * 16;
  Shared* sh = reinterpret_cast<Shared*>(satt + WARPS * ATT_PITCH);
  if (threadIdx.x == 0) sh->abort_flag = 0;
  if (threadIdx.x < 3 * 6 && (int)threadIdx.x / 6 < p.L)
    reinterpret_cast<uint4*>(sh->lw)[threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(p.layers) + threadIdx.x);
  if (p.L > 0) {                  // this warp's first attention item and the cache rows of its first keys
    constexpr int LPK = HD / 8, KPW = 32 / LPK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = 1 << p.lgw, ST = W * KPW;
    const int item = (int)blockIdx.x * (WARPS >> p.lgw) + (warp >> p.lgw), kg = (warp & (W - 1)) * KPW + lane / LPK;
    if (item < p.G * p.H) {
      const int pos = p.pos[item / p.H], slot = p.slot[item / p.H];
      if (lane == 0) { sh->item_pos[warp] = pos; sh->item_slot[warp] = slot; }
      if (lane % LPK == 0 && slot >= 0)
        for (int i = 0; i < keys_ahead<LGW, HD>(); i++) {
          const int j = kg + i * ST, jb = p.block_of(j);
          if (j < pos && jb < p.max_lb && j < p.max_ctx)
            sh->item_row[warp][lane / LPK][i] = p.btab[(size_t)slot * p.max_lb + jb] * p.bs + (j - jb * p.bs);
        }
    }
  }
  __syncthreads();
  // epochs used before this launch: constant while it runs (only its last CTA to leave advances the word)
  const uint32_t base = *reinterpret_cast<volatile uint32_t*>(p.ctl);
  const int d = p.d;
  int flip = 0;
  // the product behind a LayerNorm of half layer hl: qkv (even), fc (odd), after the last one the head
  auto ln_phase = [&](int hl) {
    Lin L;
    const int l = hl >> 1;
    const LayerW* lw = sh->lw + (l & 3);
    L.K = d; L.res = nullptr; L.e_res = 0;
    if (hl == 2 * p.L) {
      L.W = p.head_w; L.bias = nullptr; L.N = p.V; L.lgs = p.lgs_h; L.kind = PH; L.dst = nullptr;
    } else if (hl & 1) {
      L.W = lw->fc_w; L.bias = lw->fc_b; L.N = 4 * d; L.lgs = p.lgs_d; L.kind = PD; L.dst = p.actp;
    } else {
      L.W = lw->qkv_w; L.bias = lw->qkv_b; L.N = 3 * d; L.lgs = p.lgs_a; L.kind = PA; L.dst = p.qkvp;
    }
    L.src = L.kind == PD ? p.midp : (hl == 0 ? nullptr : p.xp);
    L.e_dst = base + l + 1;
    L.e_src = L.kind == PD ? L.e_dst : base + l;
    return L;
  };
  // the product that writes the residual stream in half layer hl: proj (even), fcproj (odd)
  auto res_phase = [&](int hl) {
    Lin L;
    const int l = hl >> 1;
    const LayerW* lw = sh->lw + (l & 3);
    L.N = d;
    L.e_src = L.e_dst = base + l + 1;
    if (hl & 1) {
      L.W = lw->fcproj_w; L.bias = lw->fcproj_b; L.K = 4 * d; L.lgs = p.lgs_e; L.kind = PE;
      L.src = p.actp; L.res = p.midp; L.e_res = L.e_dst; L.dst = p.xp;
    } else {
      L.W = lw->proj_w; L.bias = lw->proj_b; L.K = d; L.lgs = p.lgs_c; L.kind = PC;
      L.src = p.attp; L.res = l == 0 ? nullptr : p.xp; L.e_res = base + l; L.dst = p.midp;
    }
    return L;
  };
  const int n_half = 2 * p.L;
  // Weights go into L2 ahead of their phase: the copies into shared memory then take an L2 trip, and the memory streams during
  // attention and hand-offs too.  `far`: two phases ahead, for layers of up to 40 MB (L24 d1024: 489 -> 470 us a step at G = 1); larger
  // ones one phase ahead (L12, G = 1 / 8, one against two phases: d1280 359 / 452 and 360 / 446, d1536 390 / 502 and 397 / 518,
  // d2048 522 / 618 and 551 / 660).
  const bool far = d <= 1280;
  auto prefetch_next = [&](bool last, const LayerW* nw) {
    if (!last) {
      prefetch_units<LGW>(nw->qkv_w, 3 * d, d, (WARPS >> p.lgs_a) * 16, 8);
      prefetch_units<LGW>(nw->proj_w, d, d, (WARPS >> p.lgs_c) * 8, 8);
    } else if (p.head_w) prefetch_units<LGW>(p.head_w, p.V, d, (WARPS >> p.lgs_h) * 16, 2);
  };
  if (p.L > 0) {
    fetch_ln<LGW>(sln, sh->lw[0].ln1_w, sh->lw[0].ln1_b, d);
    prefetch_units<LGW>(sh->lw[0].proj_w, d, d, (WARPS >> p.lgs_c) * 8, 8);
  } else {
    fetch_ln<LGW>(sln, p.lnf_w, p.lnf_b, d);
  }
#pragma unroll 1
  for (int hl = 0; hl < n_half + (p.head_w ? 1 : 0); hl++) {
    const int l = hl >> 1;
    const LayerW* lw = sh->lw + (l & 3);
    const LayerW* nw = sh->lw + ((l + 1) & 3);
    const bool even = (hl & 1) == 0, last = l + 1 >= p.L;
    {
      const Lin L = ln_phase(hl);
      copy_first<LGW, 2>(wbuf, L);
      if (hl < n_half) {
        if (even) prefetch_units<LGW>(lw->fc_w, 4 * d, d, (WARPS >> p.lgs_d) * 16, 8);
        else if (far) prefetch_next(last, nw);
      }
      linear_phase<LGW, MT, true>(p, L, hl == n_half ? p.n_rows : p.G, false, xs, sln, red, flip, sh, wbuf);
    }
    if (hl == n_half) break;
    if (even) {
      // record of the layer after the next, in the place of the last one's: every warp is past the barrier of this phase, so
      // nobody reads that any more
      if (l > 0 && l + 2 < p.L) {
        const int t = tid_fresh();
        if (t < 6) cp_async16(smem_u32(reinterpret_cast<uint4*>(sh->lw + ((l + 2) & 3)) + t), reinterpret_cast<const uint4*>(p.layers + l + 2) + t);
        cp_async_commit();
      }
      if (far) prefetch_units<LGW>(lw->fcproj_w, d, 4 * d, (WARPS >> p.lgs_e) * 8, 8);
      attention_phase<LGW, HD>(p, l, base + l + 1, satt, sh);
    }
    const Lin L = res_phase(hl);
    copy_first<LGW, 1>(wbuf, L);
    const bf16 *lnw = even ? lw->ln2_w : last ? p.lnf_w : nw->ln1_w, *lnb = even ? lw->ln2_b : last ? p.lnf_b : nw->ln1_b;
    if (!far) {
      if (even) prefetch_units<LGW>(lw->fcproj_w, d, 4 * d, (WARPS >> p.lgs_e) * 8, 8);
      else prefetch_next(last, nw);
    }
    if (lnw) fetch_ln<LGW>(sln, lnw, lnb, d);
    linear_phase<LGW, MT, false>(p, L, p.G, last && !even, xs, sln, red, flip, sh, wbuf);
  }
  cp_async_wait_all();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(p.ctl + 2, 1u) == gridDim.x - 1) {
      p.ctl[1] = 0;
      p.ctl[2] = 0;
      __threadfence();
      *reinterpret_cast<volatile uint32_t*>(p.ctl) = base + (uint32_t)p.L + 1u;
    }
  }
}

constexpr int smem_bytes(int MT, int d) {
  const int warps = MT == 1 ? 1 << lg_warps<1>() : 1 << lg_warps<2>();
  return (MT == 1 ? 2 : 1) * (int)WBUF + 8 * MT * (d + PAD) * 2 + 4 * d + (MT == 4 ? 1 : 2) * warps * 8 * MT * 16 * 4 + warps * ATT_PITCH * 4 + (int)sizeof(Shared);
}
static_assert(smem_bytes(1, 4096) <= SMEM_LIMIT, "eight rows of every accepted width fit");
int max_mt(int d) {             // row groups of eight whose normalised rows fit into shared memory
  for (int mt = 4; mt > 1; mt >>= 1)
    if (smem_bytes(mt, d) <= SMEM_LIMIT) return mt;
  return 1;
}
// Warps that share a unit of 8 `rg` columns.  Slices are whole 32-column steps and at most one sub-step wide where the warps
// allow it; beyond that the split grows as long as the units still fit the same number of turns of the grid, so that a narrow
// product (proj, fcproj) runs on more CTAs with less to fetch per warp.
int pick_lgs(int N, int K, int rg, int lgw, int grid) {
  const int units = (N + 8 * rg - 1) / (8 * rg), sub = (128 >> lgw) / rg * 32;
  auto fits = [&](int lg) { return (K / 32) % (1 << lg) == 0; };
  auto turns = [&](int lg) { const long per = (long)grid * ((1 << lgw) >> lg); return (units + per - 1) / per; };
  int lg = 0;
  while (lg < lgw && fits(lg + 1) && (K >> lg) > sub) lg++;
  while (lg < lgw && fits(lg + 1) && turns(lg + 1) == turns(lg)) lg++;
  return lg;
}

template <int MT, int HD>
int launch(DecodeParams& p, int grid, cudaStream_t st) {
  const int lgw = lg_warps<MT>(), d = p.d, smem = smem_bytes(MT, d);
  p.lgs_a = pick_lgs(3 * d, d, 2, lgw, grid); p.lgs_c = pick_lgs(d, d, 1, lgw, grid); p.lgs_d = pick_lgs(4 * d, d, 2, lgw, grid);
  p.lgs_e = pick_lgs(d, 4 * d, 1, lgw, grid); p.lgs_h = p.head_w ? pick_lgs(p.V, d, 2, lgw, grid) : 0;
  p.lgw = lgw;                                  // as many warps per (sequence, head) as keep all items in one turn
  while (p.lgw > 0 && (long)p.G * p.H << p.lgw > (long)grid << lgw) p.lgw--;
  cudaError_t e = cudaFuncSetAttribute(decode_layers_k<MT, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { kh_set_error("decode_layers: shared memory opt-in failed: %s", cudaGetErrorString(e)); return -1; }
  // cooperative launch: the driver guarantees that all CTAs are resident together (or refuses the launch)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(32 << lgw); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, decode_layers_k<MT, HD>, p);
  if (e != cudaSuccess) { kh_set_error("decode_layers launch failed: %s", cudaGetErrorString(e)); return -1; }
  return 0;
}
template <int HD>
int launch_rows(DecodeParams& p, int rows, int grid, cudaStream_t st) {
  if (rows <= 8) return launch<1, HD>(p, grid, st);
  if (rows <= 16) return launch<2, HD>(p, grid, st);
  return launch<4, HD>(p, grid, st);
}
int launch_any(DecodeParams& p, int rows, int grid, cudaStream_t st) {
  if (p.hd == 128) return launch_rows<128>(p, rows, grid, st);
  if (p.hd == 64) return launch_rows<64>(p, rows, grid, st);
  return launch_rows<32>(p, rows, grid, st);
}

}  // namespace

// The decode batch sizes and model shapes the persistent decode kernel accepts.
extern "C" int kh_decode_layers_ok(int G, int d, int H, int hd, int max_ctx) {
  return G >= 1 && G <= MAX_ROWS && d >= 256 && d <= 4096 && d % 256 == 0 && H * hd == d && (hd == 32 || hd == 64 || hd == 128) &&
         max_ctx >= 1 && max_ctx <= 32768;
}

// Sequences of width d that one launch holds (more run in groups, and every group reads all weights again).
extern "C" int kh_decode_layers_rows(int d) { return 8 * max_mt(d); }

// Bytes of the packet workspace (zero-initialised once, then only used by launches that follow one another).
extern "C" long kh_decode_layers_work_bytes(int d) { return 64 + (long)MAX_ROWS * 10 * (d / 2) * 8; }

// x [G, d] holds the embedded tokens on entry and the last layer's output on return.  `layers`: device
// array of L records of twelve bf16 pointers (ln1_w, ln1_b, qkv_w, qkv_b, proj_w, proj_b, ln2_w, ln2_b,
// fc_w, fc_b, fcproj_w, fcproj_b).  With `head_w` ([V, d]) the kernel also writes
// logits[i, :V] = LNf(x[rows[i]]) head_w^T for i < n_rows (row pitch ld_logits).  `work`: the packet workspace,
// not used by anything else in flight.  Rows whose normalised copies do not fit into shared memory together
// run in groups, one launch after the other.  Returns 0 or -1.
extern "C" int kh_decode_layers(void* x, const void* layers, int L, int G, int d, int H, int hd, void* kc, void* vc,
                                long layer_elems, const void* pos, const void* slot, const void* btab, int max_lb, int bs,
                                int max_ctx, float scale, const void* head_w, const void* lnf_w, const void* lnf_b,
                                void* logits, int ld_logits, int V, const void* rows, int n_rows, void* work, void* stream) {
  if (!kh_decode_layers_ok(G, d, H, hd, max_ctx)) { kh_set_error("decode_layers: unsupported shape G=%d d=%d H=%d hd=%d", G, d, H, hd); return -1; }
  if (head_w && (!lnf_w || !lnf_b || !logits || !rows || n_rows < 1 || n_rows > MAX_ROWS || V < 1 || ld_logits < V)) {
    kh_set_error("decode_layers: incomplete head arguments");
    return -1;
  }
  if (!work || ((uintptr_t)work & 15)) { kh_set_error("decode_layers: workspace missing or misaligned"); return -1; }
  int dev = 0, grid = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&grid, cudaDevAttrMultiProcessorCount, dev);      // one CTA per SM
  if (grid < 1) { kh_set_error("decode_layers: no device"); return -1; }
  DecodeParams p = {};
  p.d = d; p.H = H; p.hd = hd; p.bs = bs; p.max_lb = max_lb; p.max_ctx = max_ctx;
  p.layers = (const LayerW*)layers;
  p.kc = (bf16*)kc; p.vc = (bf16*)vc; p.layer_elems = (size_t)layer_elems;
  p.btab = (const int*)btab;
  p.ctl = (uint32_t*)work;
  const size_t row2 = (size_t)d / 2 * MAX_ROWS;
  p.xp = (uint64_t*)((uint8_t*)work + 64); p.midp = p.xp + row2; p.attp = p.midp + row2; p.qkvp = p.attp + row2; p.actp = p.qkvp + 3 * row2;
  p.bs_mul = bs > max_ctx ? 0u : (uint32_t)(((1ull << 32) + bs - 1) / bs);
  p.scale = scale;
  p.wait_ns = KH_WAIT_LIMIT_NS;
  p.err = kh_error_word_dev();
  cudaStream_t st = (cudaStream_t)stream;
  const int cap = 8 * max_mt(d);
  auto set_head = [&](int r0, int n) {
    p.head_w = (const bf16*)head_w; p.lnf_w = (const bf16*)lnf_w; p.lnf_b = (const bf16*)lnf_b;
    p.logits = (bf16*)logits + (size_t)r0 * ld_logits; p.ld_logits = ld_logits; p.V = V;
    p.rows = (const int*)rows + r0; p.n_rows = n;
  };
  const bool together = G <= cap && (!head_w || n_rows <= cap);
  for (int g0 = 0; g0 < G; g0 += cap) {
    const int n = G - g0 < cap ? G - g0 : cap;
    p.G = n; p.L = L;
    p.x = (bf16*)x + (size_t)g0 * d; p.pos = (const int*)pos + g0; p.slot = (const int*)slot + g0;
    if (head_w && together) set_head(0, n_rows);
    if (launch_any(p, head_w && together && n_rows > n ? n_rows : n, grid, st)) return -1;
  }
  if (head_w && !together) {
    for (int r0 = 0; r0 < n_rows; r0 += cap) {
      const int n = n_rows - r0 < cap ? n_rows - r0 : cap;
      p.G = n; p.L = 0; p.x = (bf16*)x;
      set_head(r0, n);
      if (launch_any(p, n, grid, st)) return -1;
    }
  }
  return 0;
}
