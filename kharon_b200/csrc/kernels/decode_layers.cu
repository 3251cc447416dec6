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
// Links.  What bounds the step is the trip from the CTAs that write an activation to those that read it (about 850 cycles
// from store to successful poll) and the instructions between two trips.  There is no grid barrier: activations are 32-bit words
// of two bf16 columns in a workspace whose empty words are zero, and a reader polls the words that it needs until none of
// them is zero (a result of two +0.0 is written as {-0.0, +0.0}).  A word is a single-copy atomic unit, so a word that is not zero
// is the result; there are no flags and no extra bytes.  The words are laid out so that a 128-byte line has
// one writer (word_at).  Every activation has four slots that the layers use in turn.  A slot's second use:
//  - when a CTA is done with layer m - SLOTS + 1, a helper warp empties the words that it will write in layer m (last used at m - SLOTS;
//    whoever has seen all inputs of a phase at m - SLOTS + 1 knows that the readers of its own outputs of the layer before are done, since every output of
//    a phase depends on all outputs of the one before);
//  - the helpers count each other (a release and an acquire at a global word) and hand the outcome to their own CTA's computing warps, which wait for
//    it before layer m.  It has been there for a layer or two by then, and those warps execute no fence, which would cost
//    each of them 0.5 to 1 us a layer (with the stores of a phase in flight; L12 d1024 G = 1 203 us a step with one, 184 so).
// Every CTA waits so before every layer, also one that takes part in the head alone (a width of 256 has 96, 32 and 128 groups of rows for 148
// CTAs): it comes to the last layer's output when that is all that can be there.
// Launches alternate between two halves of the workspace and empty the other half for the next launch, which also
// repairs what a launch that gave up has left.
//
// Weights.  Rows of a weight matrix come in groups of eight; a CTA owns a contiguous share of the groups of every product.  A
// producer warp streams them in the order of use, chunks of eight rows x 1024 columns, with bulk copies through a ring
// that fills the shared memory (12 chunks at d = 1024: about a layer ahead), so neither HBM latency nor copy instructions
// are in the chain (cp.async by the computing warps cost them 900-1500 cycles a phase, ahead of the first poll).
//
// Products.  Eight warps split K: warp w takes columns 32 (8 s + w) ... + 31 for s = 0, 1, ..., and multiplies all rows of a chunk.
// Each lane polls exactly the 16 bytes (row lane / 4, eight columns) that are its operand fragment of mma.sync m16n8k16: for
// proj and fcproj an activation goes from L2 to the tensor cores through registers, in front of a LayerNorm it passes through
// shared memory, where a warp normalises a row.  The K order inside a 32-wide step is permuted identically for both operands.  The
// weight fragments of the first chunks are in registers before the input arrives.  Up to eight sequences: weights as the
// 16-row operand (two groups), else sequences.  tcgen05's 128-row tiles, TMEM round trip and operand staging are the latency
// that this kernel exists to avoid.  Partial sums of the warps meet in shared memory and are added in warp order.
//
// Attention.  W warps share a (sequence, head) item; the four lanes of a group hold the keys and values of a position in
// 16-byte pieces that are operand fragments of the score product (mma.sync, the query as all eight columns); probabilities and
// outputs stay fp32 on the CUDA cores, a running softmax per lane group merged once.  The first keys and values of every
// group are requested before the query is polled (cached positions do not depend on this step), those of the next layer
// are prefetched into L2.
//
// Every wait is bounded: status code 9 in the library error word.
//
// Measured (L24 d1024 V50257, a captured step with embedding and sampler, on one part; in brackets epoch-tagged 8-byte packets, cp.async weights and
// rows of activations, the form before): context 160, G = 1 / 8 / 16 374 / 407 / 562 us (463 / 515 / 734), context 200, G = 32 936 (1213); L24 d2048
// context 300, G = 4 956 (1182); L8 d4096 context 200, G = 8 1070 (1603); L4 d256 G = 1 53 (57).  Of the 28 000 cycles of a layer at G = 1, 1000 each are the trips, 2000 a
// LayerNorm, 900 the products of qkv and fc, 1500 those of fcproj, 6000 the attention, 600 each the sums and epilogues.
// Numerics follow the five-kernel path: bf16 activations between phases, fp32 accumulation, GELU applied to the bf16-rounded
// pre-activation.
#include "common.cuh"

namespace {

// Eight computing warps, and a warpgroup of helpers: a producer of weights, a warp that empties activation words, two that empty the
// other half of the workspace.  With setmaxnreg the computing warps get the registers that the helpers do not need (256 x 232 + 128 x 40
// = 384 x 168).
constexpr int NW = 8, CT = NW * 32, THREADS = CT + 128;
constexpr int KC = 1024;                      // columns of a chunk: four 32-column steps of every warp
constexpr int PITCH = KC * 2 + 64;            // bytes between its rows (conflict-free fragments)
constexpr int SLOT = 8 * PITCH;
constexpr int MAX_SLOTS = 13;
constexpr int MAX_ROWS = 32;
constexpr int ATT_PITCH = 128 + 4;            // floats per warp of the attention hand-off: 128 outputs, maximum, sum
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr uint32_t POLL_LIMIT = 1u << 23;     // rounds of an L2 load, 290 cycles and more: 1.3 s at least

// Thread index, read anew in every phase: index arithmetic derived from it would otherwise be kept in registers across the layer loop.
__device__ __forceinline__ int tid_fresh() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// A value that the compiler must not carry (with all that follows from it) across the phases.
__device__ __forceinline__ int fresh(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

struct LayerW {               // bf16 pointers of one layer (device array, one entry per layer)
  const bf16 *ln1_w, *ln1_b, *qkv_w, *qkv_b, *proj_w, *proj_b, *ln2_w, *ln2_b, *fc_w, *fc_b, *fcproj_w, *fcproj_b;
};

struct DecodeParams {
  int G, d, H, L, bs, max_lb, max_ctx;
  int lgw;                                // log2 of the warps per attention item that keep all items in one turn
  int slots;                              // chunks in the ring
  const LayerW* layers;
  bf16* x;                                // [G, d] in: embedded tokens, out: last layer's output
  uint32_t* words;                        // activations: [2 halves][4 slots][x d/2 | mid d/2 | att d/2 | qkv 3d/2 | act 4d/2][32 rows]
  bf16 *kc, *vc;                          // [L, blocks, bs, H, hd]
  size_t layer_elems;
  const int *pos, *slot, *btab;
  // optional head: logits[g, :V] = LNf(x[rows[g]]) Whead^T
  const bf16 *head_w, *lnf_w, *lnf_b;
  bf16* logits;
  int ld_logits, V, n_rows;
  const int* rows;
  uint32_t* ctl;                          // [0] launches so far, [2] CTAs that left, [3 + half] rows that the half was last used for, [5 + half] CTAs that have emptied words for a layer, [16..] zeros
  float scale, inv_d;
  uint64_t wait_ns;
  int* err;
  uint32_t h_mul;                         // ceil(2^32 / H)
  uint32_t bs_mul;                        // ceil(2^32 / bs); 0 when one block holds every position
  __device__ __forceinline__ int seq_of(int item) const { return H == 1 ? item : (int)__umulhi((uint32_t)item, h_mul); }     // item / H
  // j / bs by multiplication: exact for j < max_ctx, since max_ctx * bs stays below 2^32
  __device__ __forceinline__ int block_of(int j) const { return bs == 1 ? j : (int)__umulhi((uint32_t)j, bs_mul); }
};
__host__ __device__ constexpr size_t slot_words(int d) { return (size_t)MAX_ROWS * 5 * d; }
constexpr int SLOTS = 4;                      // of every activation: layers that lie between two uses of a word
__host__ __device__ constexpr size_t half_words(int d) { return SLOTS * slot_words(d); }
constexpr int CTL_BYTES = 512;                // 64 bytes of counters, and zeros that stand in for cache rows that do not exist

struct Shared {               // small control block behind the data regions
  uint64_t full[MAX_SLOTS], empty[MAX_SLOTS], ln_full[2], ln_empty[2];
  int item_pos[NW], item_slot[NW], pos_row[NW];     // position, slot and cache row of each warp's first attention item (constant over the layers)
  int share[4][2];                                  // this CTA's groups of eight weight rows of 3d, d, 4d and V rows
  int item_row[NW][8][4];                           // cache rows of its first keys, per lane group
  volatile int abort_flag;
  volatile uint32_t launch;                         // launches before this one
  volatile int lgw;                                 // log2 of the warps per attention item
  volatile int phase, cleared;                      // phases that the computing warps have entered / layer whose words are empty in every CTA
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
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// rows 0..7 of the product from `a`, rows 8..15 from `b`, 32 permuted columns
__device__ __forceinline__ void mma_rows(float (&c)[4], const uint4& a, const uint4& b, const uint4& x) {
  mma_bf16(c, a.x, b.x, a.y, b.y, x.x, x.y);
  mma_bf16(c, a.z, b.z, a.w, b.w, x.z, x.w);
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {     // 16-byte aligned, multiple of 16
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CT) : "memory"); }

typedef f32x2 f2;
__device__ __forceinline__ void un8(f2* f, const uint4& v) { f[0] = un2(v.x); f[1] = un2(v.y); f[2] = un2(v.z); f[3] = un2(v.w); }
__device__ __forceinline__ f2 sum8(const uint4& v) {
  f2 f[4];
  un8(f, v);
  return add2(add2(f[0], f[1]), add2(f[2], f[3]));
}
__device__ __forceinline__ f2 dev8(const uint4& v, f2 nmean, f2 acc) {       // acc + squared deviations
  f2 f[4];
  un8(f, v);
#pragma unroll
  for (int i = 0; i < 4; i++) { const f2 t = add2(f[i], nmean); acc = fma2(t, t, acc); }
  return acc;
}
__device__ __forceinline__ uint4 norm8(const uint4& v, const uint4& gw, const uint4& gb, f2 nmean, f2 rstd) {
  auto n2 = [&](uint32_t x2, uint32_t w2, uint32_t b2) {
    const f2 y = fma2(mul2(add2(un2(x2), nmean), rstd), un2(w2), un2(b2));
    return pack_bf16(lo2(y), hi2(y));
  };
  return make_uint4(n2(v.x, gw.x, gb.x), n2(v.y, gw.y, gb.y), n2(v.z, gw.z, gb.z), n2(v.w, gw.w, gb.w));
}

// ---- bounded waits.  One that runs out sets the CTA's abort flag, which ends all others of the CTA at once; the CTAs that depend on
// this one run out by themselves.  Kept short on purpose: what a layer executes has to fit into the instruction cache.
__device__ __forceinline__ void wait_bar(uint32_t bar, uint32_t parity, Shared* sh, uint64_t limit_ns) {
  if (mbar_try(bar, parity)) return;
  const uint64_t t0 = kh_globaltimer();
#pragma unroll 1
  while (!mbar_try(bar, parity))
    if (sh->abort_flag || kh_globaltimer() - t0 > limit_ns) { sh->abort_flag = 1; return; }
}
// until the words of layer n are empty in every CTA
__device__ __forceinline__ int ld_cleared(Shared* sh) {
  int v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(const_cast<int*>(&sh->cleared))) : "memory");
  return v;
}
__device__ __forceinline__ void wait_cleared(int n, Shared* sh, uint64_t limit_ns) {
  if (ld_cleared(sh) >= n) return;
  const uint64_t t0 = kh_globaltimer();
#pragma unroll 1
  while (ld_cleared(sh) < n)
    if (sh->abort_flag || kh_globaltimer() - t0 > limit_ns) { sh->abort_flag = 1; return; }
}
// after an unsuccessful round of a poll: true when the wait is over
__device__ __forceinline__ bool expired(uint32_t& it, Shared* sh) {
  if (++it > POLL_LIMIT) sh->abort_flag = 1;
  return sh->abort_flag != 0;
}

// ---- activations
__device__ __forceinline__ uint32_t ld_word(const uint32_t* p) {
  uint32_t a;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(p) : "memory");
  return a;
}
__device__ __forceinline__ void st_word(uint32_t* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t full_word(uint32_t v) { return v == 0u ? 0x80000000u : v; }
__device__ __forceinline__ void ld_words(uint4& v, const uint32_t* p) {       // four words, 16-byte aligned
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
}
__device__ __forceinline__ uint32_t least(const uint4& v) { return min(min(v.x, v.y), min(v.z, v.w)); }
constexpr int STEP_BYTES = NW * 64;             // bytes of a row between a warp's steps
constexpr int GROUP = 32;
// Position of (row, column) in the words of an activation of width N: tiles of eight rows, in which the eight rows of eight columns are
// one 128-byte line.  Such a group belongs to one CTA: a line with several writers that others poll takes 2 us to settle (L24 d1024, from
// the last store of a residual to the first successful poll: 1.5-2.5 us in rows, 0.3-1.2 us in groups; a step of G = 8 511 us and 436).
__device__ __forceinline__ uint32_t word_at(int N, int row, int col, int pitch = GROUP) {
  return (row >> 3) * (4 * N) + (col >> 3) * pitch + (row & 7) * 4 + ((col & 7) >> 1);
}
// Words between the groups of fc's output: a CTA writes three or four neighbours of them, so that for few sequences two rows (G <= 2) or
// four (G <= 4) are enough; every reader then touches a quarter or half of the lines.
__device__ __forceinline__ int act_pitch(int G) { return G <= 2 ? 8 : G <= 4 ? 16 : GROUP; }
// Where a lane's operand fragments lie: the words of its row and eight columns in step 0 of tile 0, and the distance of steps.
struct Frags {
  const uint32_t* at;
  int step, tile;
};
// `group`: words between the groups, 0: rows [n, K] of an ordinary tensor or of the attention outputs (a head of a sequence is one CTA's)
__device__ __forceinline__ Frags frags(const uint32_t* src, int group, int K, int row, int warp, int lane) {
  Frags f;
  const int pitch = group ? group : 4;
  f.at = src + row * (group ? 4 : K / 2) + (warp * 4 + (lane & 3)) * pitch;
  f.step = NW * 4 * pitch;
  f.tile = 4 * K;
  return f;
}
// A lane's fragments of four steps; of a partial last quad (`left` < 4) the last step that exists stands in for the others.
__device__ __forceinline__ void ld_quad(uint4* v, int stride, const uint32_t* p, int step, int left) {
  const uint32_t* p1 = p + (left > 1 ? step : 0);
  const uint32_t* p2 = p1 + (left > 2 ? step : 0);
  ld_words(v[0], p); ld_words(v[stride], p1); ld_words(v[2 * stride], p2); ld_words(v[3 * stride], p2 + (left > 3 ? step : 0));
}
// Until none of the words of a quad is empty (its loads have been issued).  Lanes of rows that do not exist read the last row that does, and
// nothing is loaded conditionally: a register that one path leaves unset counts as live all the way back through the layer
// loop, and the spills that follow cost an L2 trip each (shared memory leaves no L1; L24 d1024 G = 1 708 us a step with
// them, 461 without).
__device__ __forceinline__ void poll_quad(uint4* v, int stride, const uint32_t* p, int step, int left, Shared* sh) {
  uint32_t it = 0;
#pragma unroll 1
  while (min(min(least(v[0]), least(v[stride])), min(least(v[2 * stride]), least(v[3 * stride]))) == 0u) {
    if (expired(it, sh)) break;
    ld_quad(v, stride, p, step, left);
  }
}

// ---- the five products
enum Phase { PA, PC, PD, PE, PH };
struct Lin {
  const bf16* bias;         // [N] (null for the head)
  int N, K, kind, seq;      // kind PA ... PE, PH; seq: number of the phase
  const uint32_t* src;      // words [32, K / 2] of the input (null: plain rows of p.x)
  const uint32_t* res;      // C, E: words [32, N / 2] of the residual (null: plain rows of p.x)
  uint32_t* dst;            // words [32, N / 2] of the output (null for the head)
};
constexpr int LN_GROUPS = 4;                  // groups that a turn takes behind a LayerNorm (proj and fcproj: one)
constexpr int PAD = 32;                       // bf16 elements behind a normalised row (64 bytes: conflict-free fragments)

// The ring as a warp sees it: the next chunk's slot and the parity of its barrier.
struct Ring {
  uint32_t base, full, empty, ln_full, ln_empty;
  int n, slot;
  uint32_t par;
  uint8_t* ln;              // buffers of LayerNorm gain and bias (4 d bytes each), how many, the next one and its parity
  int n_ln, ln_slot;
  uint32_t ln_par;
  __device__ __forceinline__ void ln_step() {
    if (++ln_slot == n_ln) { ln_slot = 0; ln_par ^= 1u; }
  }
  __device__ __forceinline__ void step() {
    if (++slot == n) { slot = 0; par ^= 1u; }
  }
};
// hands the last `n` chunks that were taken back to the producer
__device__ __forceinline__ void release(const Ring& r, int n, int lane) {
  __syncwarp();
  if (lane < n) {
    int s = r.slot - 1 - lane;
    if (s < 0) s += r.n;
    mbar_arrive(r.empty + 8 * s);
  }
}
constexpr int lg_rows(int MT) { return MT == 1 ? 3 : (MT == 2 ? 4 : 5); }
// Output pair o of a turn: group, row (sequence) and first column inside the group.
template <int MT>
__device__ __forceinline__ void out_pair(int o, int& g, int& row, int& c) {
  c = (o & 3) * 2;
  row = (o >> 2) & (8 * MT - 1);
  g = o >> (2 + lg_rows(MT));
}
constexpr int n_red(int MT) { return MT == 4 ? 1 : 2; }        // buffers of partial sums (shared memory for a second one lacks at 32 rows)

// Steps of a quad that exist, known at compile time where a row is one partial quad (widths below 1024: LEFT = 1, 2, 3, a LayerNorm's only quad) and
// for multiples of 1024 (LEFT = 4, every quad): without the branches of the general form (LEFT = 0) the pieces of a row are worked on together.  us a
// step, four layers, general form / this: d256 H8 G = 1 57.4 / 51.6, 32 114.5 / 96.7; d512 H8 G = 1 61.5 / 55.8, 16 83.1 / 74.0; d768 H12 G = 1
// 63.8 / 59.5, 32 139.7 / 122.5; d512 H4 G = 32 131 / 113.5.
template <int LEFT> __device__ __forceinline__ int steps_left(int st, int first) { return LEFT ? LEFT : st - first; }

// LayerNorm of rows [0, n) -> xs [8 MT][K + PAD]: the warps fetch the fragments that they will multiply, then a warp takes a row, pieces
// lane, lane + 32, ... of 16 bytes in blocks of four.
template <int MT, int LEFT>
__device__ __forceinline__ void normalise(const DecodeParams& p, const Lin& L, int n, bf16* xs, Ring& ring, Shared* sh) {
  const int tid = tid_fresh(), warp = tid >> 5, lane = tid & 31, d = L.K, st = LEFT && LEFT < 4 ? LEFT : d >> 8;
  const uint32_t pitch = (d + PAD) * 2, ln = smem_u32(ring.ln) + ring.ln_slot * (4 * d) + lane * 16;
  {
    const uint32_t to = smem_u32(xs) + (lane >> 2) * pitch + warp * 64 + (lane & 3) * 16;
    Frags f[MT];
#pragma unroll
    for (int t = 0; t < MT; t++) {
      int r = min(t * 8 + (lane >> 2), n - 1);
      if (L.kind == PH) r = __ldg(p.rows + r);
      f[t] = frags(L.src ? L.src : reinterpret_cast<const uint32_t*>(p.x), L.src ? GROUP : 0, d, L.src ? r & 7 : r, warp, lane);
      if (L.src) f[t].at += (r >> 3) * f[t].tile;
    }
#pragma unroll 1
    for (int b = 0; b < st; b += 4) {                    // all rows of a block are requested together
      uint4 v[4 * MT];
#pragma unroll
      for (int t = 0; t < MT; t++) ld_quad(v + 4 * t, 1, f[t].at, f[t].step, steps_left<LEFT>(st, b));
#pragma unroll
      for (int t = 0; t < MT; t++) {
        if (L.src) poll_quad(v + 4 * t, 1, f[t].at, f[t].step, steps_left<LEFT>(st, b), sh);
        f[t].at += 4 * f[t].step;
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (i < steps_left<LEFT>(st, b)) sts128(to + t * 8 * pitch + (b + i) * STEP_BYTES, v[4 * t + i]);
      }
    }
  }
  wait_bar(ring.ln_full + 8 * ring.ln_slot, ring.ln_par, sh, p.wait_ns);
  compute_sync();
  uint32_t row = smem_u32(xs) + warp * pitch + lane * 16;
#pragma unroll 1
  for (int r = warp; r < n; r += NW, row += NW * pitch) {
    f2 s = 0, v = 0;
    uint4 x[4];
    auto load = [&](int b) {
#pragma unroll
      for (int i = 0; i < 4; i++) x[i] = lds128(row + (b + (i < steps_left<LEFT>(st, b) ? i : 0)) * 512);
    };
    auto warp_sum = [&](float a) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      return a;
    };
    const bool one = (LEFT && LEFT < 4) || st <= 4;       // one block: it stays in registers
    load(0);
    int b = 0;
#pragma unroll 1
    do {
      if (!one) load(b);
#pragma unroll
      for (int i = 0; i < 4; i++) if (i < steps_left<LEFT>(st, b)) s = add2(s, sum8(x[i]));
    } while ((b += 4) < st);
    const float mean = warp_sum(lo2(s) + hi2(s)) * p.inv_d;
    const f2 nm = mk2(-mean, -mean);
    b = 0;
#pragma unroll 1
    do {
      if (!one) load(b);
#pragma unroll
      for (int i = 0; i < 4; i++) if (i < steps_left<LEFT>(st, b)) v = dev8(x[i], nm, v);
    } while ((b += 4) < st);
    const float rstd = rsqrtf(warp_sum(lo2(v) + hi2(v)) * p.inv_d + 1e-5f);
    const f2 rs = mk2(rstd, rstd);
    b = 0;
#pragma unroll 1
    do {
      if (!one) load(b);
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i < steps_left<LEFT>(st, b)) sts128(row + (b + i) * 512, norm8(x[i], lds128(ln + (b + i) * 512), lds128(ln + 2 * d + (b + i) * 512), nm, rs));
    } while ((b += 4) < st);
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(ring.ln_empty + 8 * ring.ln_slot);
  ring.ln_step();
}

// A product over rows [0, n), n <= 8 MT: behind a LayerNorm (A, D, head; turns of four groups) or with a residual (C, E; turns of one group).
// One copy of the code serves all phases: a layer's instructions should fit into the instruction cache (measured: straight-line
// code of up to 32 KB runs at full speed; beyond, every jump to a line that is not there costs 50 cycles, beyond 128 KB 190).
template <int MT, int LEFT>
__device__ __forceinline__ void product(const DecodeParams& p, const Lin& L, bool ln, int n, bool last, bf16* xs, float* red0, int& flip,
                                        Ring& ring, Shared* sh) {
  constexpr int MH = MT == 1 ? 1 : MT / 2;               // accumulators of a group
  constexpr int QB = 4 / MT;                             // C, E: chunks whose weights and activations are in flight together
  constexpr int NA = LN_GROUPS * MH;
  const int tid = tid_fresh(), warp = tid >> 5, lane = tid & 31;
  if (tid == 0) sh->phase = L.seq + 1;
  const int sx = L.kind == PA ? 0 : L.kind == PD ? 2 : L.kind == PH ? 3 : 1;
  const int g0 = sh->share[sx][0], g1 = sh->share[sx][1];
  if (g0 >= g1) return;                                  // uniform over the CTA
  const int st = L.K >> 8, nq = (st + 3) >> 2;           // steps of a warp and chunks of a row
  const uint32_t lane_off = ring.base + (lane >> 2) * PITCH + warp * 64 + (lane & 3) * 16;
  bool first = true;
#pragma unroll 1
  for (int t0 = g0; t0 < g1; t0 += ln ? LN_GROUPS : 1) {
    const int ng = ln ? min(LN_GROUPS, g1 - t0) : 1;
    uint32_t bias2 = 0, res2 = 0;                        // of output pair tid, as they are now
    auto operands = [&](int g, int row, int col) {
      if (L.bias) bias2 = __ldg(reinterpret_cast<const unsigned int*>(L.bias + col));
      if (!ln) {
        res2 = L.res ? ld_word(L.res + word_at(L.N, row, col)) : __ldcg(reinterpret_cast<const unsigned int*>(p.x) + (uint32_t)(row * L.N + col) / 2);
      }
    };
    {
      int g, row, c;
      out_pair<MT>(tid, g, row, c);
      if (g < ng && row < n && (t0 + g) * 8 + c < L.N) operands(g, row, (t0 + g) * 8 + c);
    }
    float acc[NA][4];
#pragma unroll
    for (int a = 0; a < NA; a++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[a][i] = 0.f;
#pragma unroll 1
    for (int q0 = 0; q0 < nq; q0 += ln ? 1 : QB) {
      const int nc = ln ? ng : min(QB, nq - q0), left = ln ? steps_left<LEFT>(st, 4 * q0) : steps_left<LEFT == 4 ? 4 : 0>(st, 4 * q0);
      uint4 x[16], w[16];                                // LN: [step][tile]; C, E: [chunk][step][tile] of QB chunks.  [chunk][step]
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const uint32_t a = lane_off + ring.slot * SLOT;
        if (c < nc) {                                    // (else: whatever is there, for rows that nobody reads)
          wait_bar(ring.full + 8 * ring.slot, ring.par, sh, p.wait_ns);
          ring.step();
        }
#pragma unroll
        for (int i = 0; i < 4; i++) w[4 * c + i] = lds128(a + i * STEP_BYTES);
      }
      if (ln) {
        if (first) {
          first = false;
          normalise<MT, LEFT>(p, L, n, xs, ring, sh);
          compute_sync();
        }
        {
          const uint32_t xa = smem_u32(xs) + (lane >> 2) * ((L.K + PAD) * 2) + warp * 64 + (lane & 3) * 16 + q0 * (4 * STEP_BYTES);
#pragma unroll
          for (int i = 0; i < 4 * MT; i++) x[i] = lds128(xa + i % MT * 16 * (L.K + PAD) + (i / MT < left ? i / MT * STEP_BYTES : 0));
        }
#pragma unroll
        for (int s = 0; s < 4; s++)
          if (s < left) {
            if constexpr (MT == 1) {      // weights of two groups are the 16 rows; two chains per pair
#pragma unroll
              for (int g = 0; g < LN_GROUPS; g += 2) {
                const uint4 w0 = w[g * 4 + s], w1 = w[g * 4 + 4 + s];
                mma_bf16(acc[g], w0.x, w1.x, w0.y, w1.y, x[s].x, x[s].y);
                mma_bf16(acc[g + 1], w0.z, w1.z, w0.w, w1.w, x[s].z, x[s].w);
              }
            } else {                      // sequences are the 16 rows
#pragma unroll
              for (int g = 0; g < LN_GROUPS; g++)
#pragma unroll
                for (int m = 0; m < MH; m++) mma_rows(acc[g * MH + m], x[s * MT + 2 * m], x[s * MT + 2 * m + 1], w[g * 4 + s]);
            }
          }
      } else {
        // ---- proj, fcproj: the fragments come straight from the words
        const int group = L.kind == PE ? act_pitch(n) : 0;
        const uint32_t* rows[MT];
        int step = 0;
#pragma unroll
        for (int t = 0; t < MT; t++) {
          const int r = min(t * 8 + (lane >> 2), n - 1);
          const Frags f = frags(L.src, group, L.K, group ? r & 7 : r, warp, lane);
          step = f.step;
          rows[t] = f.at + (group ? (r >> 3) * f.tile : 0) + q0 * 4 * step;
        }
#pragma unroll
        for (int c = 0; c < QB; c++)
#pragma unroll
          for (int t = 0; t < MT; t++)
            if (c < nc) ld_quad(x + c * 4 * MT + t, MT, rows[t] + c * 4 * step, step, steps_left<LEFT == 4 ? 4 : 0>(left, 4 * c));
            else
#pragma unroll
              for (int i = 0; i < 4; i++) x[(c * 4 + i) * MT + t] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int c = 0; c < QB; c++)
          if (c < nc) {
#pragma unroll
            for (int t = 0; t < MT; t++) poll_quad(x + c * 4 * MT + t, MT, rows[t] + c * 4 * step, step, steps_left<LEFT == 4 ? 4 : 0>(left, 4 * c), sh);
            __syncwarp();
#pragma unroll
            for (int s = 0; s < 4; s++)
              if (s < steps_left<LEFT == 4 ? 4 : 0>(left, 4 * c)) {
                const uint4 w0 = w[c * 4 + s];
                const uint4* xv = x + (c * 4 + s) * MT;
                if constexpr (MT == 1) {
                  mma_bf16(acc[(2 * s) & 3], w0.x, 0u, w0.y, 0u, xv[0].x, xv[0].y);
                  mma_bf16(acc[(2 * s + 1) & 3], w0.z, 0u, w0.w, 0u, xv[0].z, xv[0].w);
                } else {
#pragma unroll
                  for (int m = 0; m < MH; m++) {      // two chains per pair of tiles
                    mma_bf16(acc[m], xv[2 * m].x, xv[2 * m + 1].x, xv[2 * m].y, xv[2 * m + 1].y, w0.x, w0.y);
                    mma_bf16(acc[MH + m], xv[2 * m].z, xv[2 * m + 1].z, xv[2 * m].w, xv[2 * m + 1].w, w0.z, w0.w);
                  }
                }
              }
          }
      }
      release(ring, nc, lane);
    }
    // ---- partial sums -> red[warp][group][sequence][weight row]
    float* red = red0;
    if (n_red(MT) == 1) compute_sync();                   // everybody has read the previous turn's
    else { flip ^= 1; red += flip * (NW * LN_GROUPS * 64 * MT); }
    {
      float* mine = red + warp * (LN_GROUPS * 64 * MT);
      if constexpr (MT == 1) {
        mine += (lane & 3) * 16 + (lane >> 2);
        if (!ln)
#pragma unroll
          for (int i = 0; i < 2; i++) { acc[0][i] += acc[2][i]; acc[1][i] += acc[3][i]; }
#pragma unroll
        for (int g = 0; g < LN_GROUPS; g++)
          if (g < ng)
#pragma unroll
            for (int i = 0; i < 2; i++) mine[g * 64 + i * 8] = acc[g & ~1][(g & 1) * 2 + i] + acc[g | 1][(g & 1) * 2 + i];
      } else {
        mine += lane * 2;
        if (!ln)
#pragma unroll
          for (int m = 0; m < MH; m++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[m][i] += acc[MH + m][i];
#pragma unroll
        for (int g = 0; g < LN_GROUPS; g++)
          if (g < ng)
#pragma unroll
            for (int m = 0; m < MH; m++) {
              const float* c = acc[g * MH + m];
              *reinterpret_cast<float2*>(mine + g * (64 * MT) + m * 128) = make_float2(c[0], c[1]);
              *reinterpret_cast<float2*>(mine + g * (64 * MT) + m * 128 + 64) = make_float2(c[2], c[3]);
            }
      }
    }
    compute_sync();
    // ---- sum over the warps in order, epilogue, and on their way
#pragma unroll 1
    for (int o = tid; o < ng * 32 * MT; o += CT) {
      int g, row, c;
      out_pair<MT>(o, g, row, c);
      const int col = (t0 + g) * 8 + c;
      if (row >= n || col >= L.N) continue;
      if (MT > 2 && o != tid) operands(g, row, col);
      const float* t = red + g * (64 * MT) + row * 8 + c;
      const uint32_t at = word_at(L.N, row, col, L.kind == PD ? act_pitch(n) : GROUP);
      float2 f[NW];
#pragma unroll
      for (int i = 0; i < NW; i++) f[i] = *reinterpret_cast<const float2*>(t + i * (LN_GROUPS * 64 * MT));
      uint32_t it = 0;
#pragma unroll 1
      while (!ln && L.res && res2 == 0 && !expired(it, sh)) res2 = ld_word(L.res + at);
      f2 v = 0;
#pragma unroll
      for (int i = 0; i < NW; i++) v = add2(v, mk2(f[i].x, f[i].y));
      v = add2(v, un2(bias2));
      if (!ln) v = add2(v, un2(res2));
      float v0 = lo2(v), v1 = hi2(v);
      if (L.kind == PD) {
        v0 = gelu_tanh(__bfloat162float(__float2bfloat16(v0)));
        v1 = gelu_tanh(__bfloat162float(__float2bfloat16(v1)));
      }
      const uint32_t pk = pack_bf16(v0, v1);
      if (L.dst) {
        st_word(L.dst + at, full_word(pk));
        if (last) reinterpret_cast<uint32_t*>(p.x)[(uint32_t)(row * L.N + col) / 2] = pk;
      } else {
        bf16* q = p.logits + (size_t)row * p.ld_logits + col;
        if (col + 1 < L.N && ((uintptr_t)q & 3) == 0) *reinterpret_cast<uint32_t*>(q) = pk;
        else {
          q[0] = __float2bfloat16(v0);
          if (col + 1 < L.N) q[1] = __float2bfloat16(v1);
        }
      }
    }
  }
}

// ---- helpers
// Producer: the chunks of this CTA's share of W [N, K] in the order in which the computing warps take them.
__device__ __forceinline__ bool stream(const bf16* W, int N, int K, int per_turn, const int* range, Ring& r, Shared* sh, const DecodeParams& p) {
  const int lane = threadIdx.x & 31, g1 = range[1];
#pragma unroll 1
  for (int t0 = range[0]; t0 < g1; t0 += per_turn)
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += KC)
#pragma unroll 1
      for (int g = t0; g < min(t0 + per_turn, g1); g++) {
        wait_bar(r.empty + 8 * r.slot, r.par ^ 1u, sh, 2 * p.wait_ns);
        if (sh->abort_flag) return false;
        const int rows = min(8, N - g * 8), bytes = min(KC, K - k0) * 2;
        if (lane == 0) mbar_expect_tx(r.full + 8 * r.slot, rows * bytes);
        __syncwarp();
        if (lane < rows) bulk_load(r.base + r.slot * SLOT + lane * PITCH, W + (size_t)(g * 8 + lane) * K + k0, bytes, r.full + 8 * r.slot);
        r.step();
      }
  return true;
}
__device__ __forceinline__ void produce(const DecodeParams& p, Ring ring, Shared* sh) {
  const int d = p.d;
  bool ok = true;
#pragma unroll 1
  for (int k = 0; ok && k < 4 * p.L + (p.head_w ? 1 : 0); k++) {
    const int j = k & 3;
    const bool head = k == 4 * p.L;
    const bf16* const* lw = reinterpret_cast<const bf16* const*>(p.layers + (k >> 2));
    const bf16* W = head ? p.head_w : lw[j == 0 ? 2 : j == 1 ? 4 : j == 2 ? 8 : 10];
    const int* range = sh->share[head ? 3 : j == 3 ? 1 : j];
    if (!(j & 1) && range[0] < range[1]) {               // gain and bias of the LayerNorm in front
      wait_bar(ring.ln_empty + 8 * ring.ln_slot, ring.ln_par ^ 1u, sh, 2 * p.wait_ns);
      if (sh->abort_flag) { ok = false; break; }
      if ((threadIdx.x & 31) == 0) {
        const uint32_t bar = ring.ln_full + 8 * ring.ln_slot, dst = smem_u32(ring.ln + ring.ln_slot * (4 * d));
        mbar_expect_tx(bar, 4 * d);
        bulk_load(dst, head ? p.lnf_w : lw[j ? 6 : 0], 2 * d, bar);
        bulk_load(dst + 2 * d, head ? p.lnf_b : lw[j ? 7 : 1], 2 * d, bar);
      }
      ring.ln_step();
    }
    ok = stream(W, head ? p.V : j == 0 ? 3 * d : j == 2 ? 4 * d : d, j == 3 ? 4 * d : d, j & 1 ? 1 : LN_GROUPS, range, ring, sh, p);
  }
  // No copy may be in flight when the CTA leaves, not even where all have been issued and computing warps gave up before they took them: every
  // slot's last copy is waited for, backwards over the rings (a slot that was never filled passes at once).
#pragma unroll 1
  for (int k = 0; k < ring.n_ln; k++) {
    if (ring.ln_slot == 0) { ring.ln_slot = ring.n_ln; ring.ln_par ^= 1u; }
    ring.ln_slot--;
    const uint64_t t0 = kh_globaltimer();
    while (!mbar_try(ring.ln_full + 8 * ring.ln_slot, ring.ln_par) && kh_globaltimer() - t0 < 100000000ull) {}
  }
#pragma unroll 1
  for (int k = 0; k < ring.n; k++) {
    if (ring.slot == 0) { ring.slot = ring.n; ring.par ^= 1u; }
    ring.slot--;
    const uint64_t t0 = kh_globaltimer();
    while (!mbar_try(ring.full + 8 * ring.slot, ring.par) && kh_globaltimer() - t0 < 100000000ull) {}
  }
}
// Empties this CTA's words of layer m, where layer m - SLOTS has used them, and waits for the other CTAs to have done so.
template <int HD>
__device__ __forceinline__ void empty_words(const DecodeParams& p, uint32_t* words, Shared* sh) {
  const int lane = threadIdx.x & 31;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int m = SLOTS; m < p.L; m++) {
    uint64_t t0 = kh_globaltimer();
    while (sh->phase <= 5 * (m - SLOTS + 2)) {           // until the CTA has entered the layer after m - SLOTS + 1
      if (sh->abort_flag || kh_globaltimer() - t0 > 2 * p.wait_ns) { sh->abort_flag = 1; return; }
      __nanosleep(50);
    }
    const int d = fresh(p.d), row = MAX_ROWS * (d / 2);
    uint32_t* const nxt = words + m % SLOTS * (uint32_t)slot_words(d);
    {
      const int per = NW >> sh->lgw, items = p.G * p.H;
      uint32_t* a = nxt + 2 * row;
#pragma unroll 1
      for (int it0 = (int)blockIdx.x * per; it0 < items; it0 += (int)gridDim.x * per)
#pragma unroll 1
        for (int i = lane; i < per * (HD / 8); i += 32) {
          const int it = it0 + i / (HD / 8), t = p.seq_of(it);
          if (it < items) *reinterpret_cast<uint4*>(a + (t * d + (it - t * p.H) * HD) / 2 + (i % (HD / 8)) * 4) = zero;
        }
    }
#pragma unroll 1
    for (int j = 0; j < 4; j++) {              // qkv, mid, act, x
      const int N = j == 0 ? 3 * d : j == 2 ? 4 * d : d;
      uint32_t* a = nxt + (j == 0 ? 3 : j == 1 ? 1 : j == 2 ? 6 : 0) * row;
      const int* range = sh->share[j == 0 ? 0 : j == 2 ? 2 : 1];
      const int pitch = j == 2 ? act_pitch(p.G) : GROUP;
#pragma unroll 1
      for (int r = 0; r < p.G; r += 8)
#pragma unroll 1
        for (int i = range[0] * pitch + lane * 4; i < range[1] * pitch; i += 128) *reinterpret_cast<uint4*>(a + r / 8 * (4 * N) + i) = zero;
    }
    __syncwarp();
    // Nobody counts for layer m + 1 before all have for m, so that one counter serves all layers
    uint32_t* const count = p.ctl + 5 + (sh->launch & 1u);
    if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    t0 = kh_globaltimer();
    while (true) {
      uint32_t n;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(count) : "memory");
      if (n >= gridDim.x * (uint32_t)(m - SLOTS + 1)) break;
      if (sh->abort_flag || kh_globaltimer() - t0 > 2 * p.wait_ns) { sh->abort_flag = 1; return; }
      __nanosleep(100);
    }
    __syncwarp();
    if (lane == 0) asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(smem_u32(const_cast<int*>(&sh->cleared))), "r"(m) : "memory");
  }
}
// The other half of the workspace is emptied for the next launch.
__device__ __forceinline__ void empty_half(const DecodeParams& p, uint32_t half) {
  const int used = min((int)*reinterpret_cast<volatile uint32_t*>(p.ctl + 3 + (half ^ 1u)) + 7 & ~7, MAX_ROWS), d = p.d;
  const int me = (int)blockIdx.x * 64 + (int)threadIdx.x % 64, all = (int)gridDim.x * 64;
  uint32_t* w = p.words + (half ^ 1u) * half_words(d);
#pragma unroll 1
  for (int s = 0; s < SLOTS; s++)
#pragma unroll 1
    for (int f = 0; f < 5; f++) {
      const int width = (f < 3 ? d : (f == 3 ? 3 * d : 4 * d)) / 2, from = f < 4 ? f * d / 2 : 3 * d;
      uint4* q = reinterpret_cast<uint4*>(w + s * slot_words(d) + (size_t)MAX_ROWS * from);
#pragma unroll 1
      for (int i = me; i < used * width / 4; i += all) q[i] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// log2 of the warps per attention item (whole warp, the same in every CTA).  All items in one turn leave many CTAs without one where they do not
// divide well (G = 24, 16 heads: 96 of 148 with two warps to an item); more warps to an item then take less time over long contexts, in spite of
// what a turn costs beside its positions, which is what a warp does in 30 of them.
__device__ __forceinline__ int item_warps(const DecodeParams& p) {
  const int lane = threadIdx.x & 31, items = p.G * p.H;
  int far = lane < p.G ? p.pos[lane] : 0;
  far = min(__reduce_max_sync(0xffffffffu, far), p.max_ctx);
  int best = p.lgw, cost = 0x7fffffff;
#pragma unroll 1
  for (int lg = p.lgw; lg <= 3; lg++) {
    const int per = (int)gridDim.x * (NW >> lg), c = (items + per - 1) / per * (30 + (far >> lg));
    if (c < cost) { cost = c; best = lg; }
  }
  return best;
}
// ------------------------------------------------------------------------------------------------
// Positions that a lane group (four lanes) holds at a time: the 16 rows of a score product; twice as many for many sequences with narrow heads,
// whose rows are short (L4 d512 H16 G = 32, contexts of 20 / 200 / 900: 116 / 131 / 194 us a step, 105 / 125 / 216 with two; d256 H8 100 / 108 /
// 135 and 93 / 103 / 142), and for such heads in models of long contexts (L4 d512 H16, G = 1 at 20 / 1000 / 4000 / 16000 positions 57 / 76 / 156 / 507 us with
// two, 59 / 73 / 131 / 391 with four), but not elsewhere (head width 64, L12 d1024 G = 8, 160: 205 us with two, 222 with four; L4 G = 8, 16000: 839
// and 824).
constexpr int LONG_CTX = 2048;
// Bytes of a layer's keys and values up to which the next layer's are prefetched into L2; beyond, they are gone before they are used and
// come from memory twice (G = 32, 900 positions, 118 MB: L12 d1024 977 us with, 889 without; 59 MB, G = 16: 492 and 500; 65 MB, L4 d2048 G = 8: 252 and 240).
constexpr float FETCH_LIMIT = 60e6f;
// Phase B.  Appends the new k, v to the paged cache and attends over positions 0..pos.
// The W warps of an item hold 8 W lane groups; group i takes positions i, i + 8 W, i + 16 W, ...; the group that would take `pos` starts with
// the new key and value.
template <int MT, int HD, int NB>
__device__ __forceinline__ void attention_phase(const DecodeParams& p, int layer, int seq, const uint32_t* qkvw, uint32_t* attw, float* satt, Shared* sh) {
  constexpr int NC = HD / 32;      // 16-byte pieces of a row per lane
  const int tid = tid_fresh(), warp = tid >> 5, lane = tid & 31, lgw = sh->lgw, H = fresh(p.H), bid = fresh(blockIdx.x);
  if (tid == 0) sh->phase = seq + 1;
  const int W = 1 << lgw, slots = NW >> lgw, ST = W * 8;
  const int first = (warp & (W - 1)) * 8, kg = first + (lane >> 2), e0 = (lane & 3) * 8;       // (first: uniform over the warp)
  const int d = fresh(p.d), items = p.G * H;
#pragma unroll 1
  for (int it0 = bid * slots; it0 < items; it0 += (int)gridDim.x * slots) {
    const int item = it0 + (warp >> lgw);
    const int t = p.seq_of(item), h = item - t * H;
    int pos = -1, slot = -1;
    const bool turn0 = it0 == bid * slots;
    if (item < items) {
      pos = turn0 ? sh->item_pos[warp] : __ldg(p.pos + t);
      slot = turn0 ? sh->item_slot[warp] : __ldg(p.slot + t);
    }
    const bool valid = pos >= 0 && pos < p.max_ctx && p.block_of(pos) < p.max_lb && slot >= 0;       // uniform over the item's warps
    if (item < items && !valid && lane == 0) atomicCAS(p.err, 0, 8);
    float m = -INFINITY, l = 0.f;
    f2 o[4 * NC];
#pragma unroll
    for (int k = 0; k < 4 * NC; k++) o[k] = 0;
    if (valid) {
      const int* bt = p.btab + (size_t)slot * p.max_lb;
      auto row_of = [&](int j) {
        const int jb = p.block_of(j);
        return __ldg(bt + jb) * p.bs + (j - jb * p.bs);
      };
      const int at = h * HD + e0;
      // this lane asks L2 for a line of the next layer, while a layer's keys and values (as many for all sequences as for this one) stay there until then
      const bool fetch = (lane & 3) < (HD == 128 ? 2 : 1) && layer + 1 < p.L && (float)pos * (float)(p.G * d) < FETCH_LIMIT / 4.f;
      const bf16 *kc = p.kc + (size_t)layer * p.layer_elems + at, *vc = p.vc + (size_t)layer * p.layer_elems + at;
      const bf16* none = reinterpret_cast<const bf16*>(p.ctl + 16) + e0;       // zeros, for positions that do not exist
      const bf16* vp[NB];              // this group's next values
      int row[NB];                     // cache rows of its next positions; the block table is read a turn ahead
#pragma unroll
      for (int i = 0; i < NB; i++) {
        row[i] = 0;
        if (kg + i * ST < pos) row[i] = turn0 ? sh->item_row[warp][lane >> 2][i] : row_of(kg + i * ST);
      }
      uint4 k4[NB][NC], v4[NB][NC];    // refilled with the next positions as soon as they are used
      uint4 q[NC];
#pragma unroll
      for (int k = 0; k < NC; k++) {
        q[k] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < NB; i++) k4[i][k] = v4[i][k] = make_uint4(0u, 0u, 0u, 0u);
      }
      // Turn -1 only requests the first NB keys and values and then waits for the query; every other turn uses NB positions
      // and requests the next ones in their place.
#pragma unroll 1
      for (int b0 = -NB * ST; b0 < 0 || first + b0 < pos; b0 += NB * ST) {
        const int jn = kg + b0 + NB * ST;
        float s[NB];
        int e[NB];
#pragma unroll
        for (int i = 0; i < NB; i++) {
          s[i] = 0.f;
          e[i] = 0;
          if (jn + (NB + i) * ST < pos) e[i] = __ldg(bt + p.block_of(jn + (NB + i) * ST));
        }
        if (b0 >= 0) {
#pragma unroll
          for (int i = 0; i < NB; i += 2) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < NC; k++) mma_rows(c, k4[i][k], k4[i + 1][k], q[k]);
            s[i] = c[0]; s[i + 1] = c[2];
          }
        }
        // cached positions only; the same lines of the next layer are requested into L2
#pragma unroll
        for (int i = 0; i < NB; i++) {
          const bool in = jn + i * ST < pos;
          const bf16* kp = none;
          vp[i] = none;
          if (in) {
            const size_t r = (size_t)(uint32_t)row[i] * (uint32_t)d;
            kp = kc + r;
            vp[i] = vc + r;
            if (fetch) { prefetch_l2(kp + p.layer_elems + e0 * 7); prefetch_l2(vp[i] + p.layer_elems + e0 * 7); }
          }
#pragma unroll
          for (int k = 0; k < NC; k++) k4[i][k] = ldg_stream(kp + k * 32);
        }
        if (b0 >= 0) {
          float mn = m;
#pragma unroll
          for (int i = 0; i < NB; i++) {
            s[i] = kg + b0 + i * ST < pos ? s[i] * p.scale : -INFINITY;
            mn = fmaxf(mn, s[i]);
          }
          const float ref = mn == -INFINITY ? 0.f : mn, sc = __expf(m - ref);
          m = mn;
          l *= sc;
#pragma unroll
          for (int k = 0; k < 4 * NC; k++) o[k] = mul2(o[k], mk2(sc, sc));
#pragma unroll
          for (int i = 0; i < NB; i++) {
            const float pr = __expf(s[i] - ref);
            l += pr;
#pragma unroll
            for (int k = 0; k < NC; k++) {
              f2 f[4];
              un8(f, v4[i][k]);
#pragma unroll
              for (int e = 0; e < 4; e++) o[4 * k + e] = fma2(mk2(pr, pr), f[e], o[4 * k + e]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < NB; i++)
#pragma unroll
          for (int k = 0; k < NC; k++) v4[i][k] = ldg_stream(vp[i] + k * 32);
        if (b0 < 0) {
          const uint32_t* qp = qkvw + word_at(3 * d, t, at);        // (32 columns are 128 words on)
          const bool owner = (pos & (ST - 1)) == kg;
          uint4 kn[NC], vn[NC];
#pragma unroll
          for (int k = 0; k < NC; k++) kn[k] = vn[k] = make_uint4(0u, 0u, 0u, 0u);
          uint32_t it = 0;
#pragma unroll 1
          while (true) {
            uint32_t e = 0xffffffffu;
#pragma unroll
            for (int k = 0; k < NC; k++) ld_words(q[k], qp + 128 * k);
            if (owner) {
#pragma unroll
              for (int k = 0; k < NC; k++) { ld_words(kn[k], qp + 4 * d + 128 * k); ld_words(vn[k], qp + 8 * d + 128 * k); }
#pragma unroll
              for (int k = 0; k < NC; k++) e = min(e, min(least(kn[k]), least(vn[k])));
            }
#pragma unroll
            for (int k = 0; k < NC; k++) e = min(e, least(q[k]));
            if (e != 0u || expired(it, sh)) break;
          }
          __syncwarp();
          float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int k = 0; k < NC; k++) mma_rows(c, kn[k], make_uint4(0u, 0u, 0u, 0u), q[k]);
          if (owner) {
            m = c[0] * p.scale;
            l = __expf(m - (m == -INFINITY ? 0.f : m));
            const size_t dst = (size_t)(uint32_t)(turn0 ? sh->pos_row[warp] : row_of(pos)) * (uint32_t)d;
#pragma unroll
            for (int k = 0; k < NC; k++) {
              f2 f[4];
              un8(f, vn[k]);
#pragma unroll
              for (int e = 0; e < 4; e++) o[4 * k + e] = mul2(mk2(l, l), f[e]);
              *reinterpret_cast<uint4*>(const_cast<bf16*>(kc) + dst + k * 32) = kn[k];
              *reinterpret_cast<uint4*>(const_cast<bf16*>(vc) + dst + k * 32) = vn[k];
            }
          }
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
          const int j = jn + (NB + i) * ST;
          row[i] = e[i] * p.bs + (j - p.block_of(j) * p.bs);
        }
      }
      __syncwarp();
    } else { m = 0.f; l = 0.125f; }    // an item with a bad index writes zeros: its row must not stall
    // merge the lane groups of the warp: every round adds half of the values of the partner and gives it the other half
    float mx = m;
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
    const float c = __expf(m - (mx == -INFINITY ? 0.f : mx));
    l *= c;
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
    float v[8 * NC];
#pragma unroll
    for (int k = 0; k < 4 * NC; k++) { v[2 * k] = lo2(o[k]) * c; v[2 * k + 1] = hi2(o[k]) * c; }
    int f0 = 0;
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const int x = 16 >> r, half = (4 * NC) >> r;
      const bool up = (lane & x) != 0;
      if (up) f0 += half;
#pragma unroll
      for (int i = 0; i < half; i++) {
        const float give = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, x);
      }
    }
    float* mine = satt + warp * ATT_PITCH;
#pragma unroll
    for (int i = 0; i < NC; i++) mine[((f0 + i) >> 3) * 32 + e0 + ((f0 + i) & 7)] = v[i];
    if (lane == 0) *reinterpret_cast<float2*>(mine + 128) = make_float2(mx, l);
    compute_sync();
    // merge the W warps of each item
#pragma unroll 1
    for (int i = tid; i < slots * (HD / 2); i += CT) {
      const int sl = i / (HD / 2), e = (i % (HD / 2)) * 2, it = it0 + sl;
      const float* part = satt + (size_t)(sl << lgw) * ATT_PITCH;
      float top = -INFINITY;
#pragma unroll 4
      for (int k = 0; k < W; k++) top = fmaxf(top, part[k * ATT_PITCH + 128]);
      float den = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll 4
      for (int k = 0; k < W; k++) {
        const float2 ml = *reinterpret_cast<const float2*>(part + k * ATT_PITCH + 128), f = *reinterpret_cast<const float2*>(part + k * ATT_PITCH + e);
        const float ck = __expf(ml.x - top);           // (NaN when every score is -inf, as in the kernel chain)
        den += ck * ml.y;
        v0 += ck * f.x; v1 += ck * f.y;
      }
      const float inv = 1.f / den;
      const int tt = p.seq_of(it);
      if (it < items) st_word(attw + ((size_t)tt * d + (it - tt * H) * HD + e) / 2, full_word(pack_bf16(v0 * inv, v1 * inv)));
    }
    compute_sync();                // satt is reused by the next turn or layer
  }
}

__host__ __device__ constexpr int n_ln(int d) { return d <= 1536 ? 2 : 1; }     // buffers of LayerNorm gain and bias (wide models: the ring is no deeper than a phase)

template <int MT, int HD, int NB, int LEFT>
__global__ void __launch_bounds__(THREADS, 1) decode_layers_k(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int d = p.d;
  uint8_t* at = smem + p.slots * SLOT;
  bf16* xs = reinterpret_cast<bf16*>(at);
  at += 16 * MT * (d + PAD);
  uint8_t* sln = at;
  at += n_ln(d) * 4 * d;
  float* red = reinterpret_cast<float*>(at);
  at += n_red(MT) * NW * LN_GROUPS * 64 * MT * 4;
  float* satt = reinterpret_cast<float*>(at);
  at += NW * ATT_PITCH * 4;
  Shared* sh = reinterpret_cast<Shared*>(at);

  const int warp = threadIdx.x >> 5;
  Ring ring = {smem_u32(smem), smem_u32(sh->full), smem_u32(sh->empty), smem_u32(sh->ln_full), smem_u32(sh->ln_empty), p.slots, 0, 0u, sln, n_ln(d), 0, 0u};
  if (threadIdx.x == 0) {
    sh->abort_flag = 0;
    sh->phase = 0;
    sh->cleared = SLOTS - 1;             // (the launch starts with empty slots)
    for (int s = 0; s < p.slots; s++) { mbar_init(ring.full + 8 * s, 1); mbar_init(ring.empty + 8 * s, NW); }
    for (int s = 0; s < 2; s++) { mbar_init(ring.ln_full + 8 * s, 1); mbar_init(ring.ln_empty + 8 * s, NW); }
    mbar_fence_init();
  }
  if (threadIdx.x < 8) {
    const int k = (int)threadIdx.x >> 1, e = (int)threadIdx.x & 1;
    const unsigned groups = (unsigned)(k == 0 ? 3 * d : k == 1 ? d : k == 2 ? 4 * d : p.V + 7) / 8;
    sh->share[k][e] = (int)(groups * (blockIdx.x + e) / gridDim.x);
  }
  // launches before this one: constant while it runs (only its last CTA to leave advances the word)
  if (threadIdx.x == 0) sh->launch = *reinterpret_cast<volatile uint32_t*>(p.ctl);
  if (warp == 1 && p.L > 0) sh->lgw = item_warps(p);      // (a launch for the head alone has no positions)
  __syncthreads();

  if (warp >= NW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    const uint32_t half = sh->launch & 1u;
    if (warp == NW) produce(p, ring, sh);
    else if (warp == NW + 1) empty_words<HD>(p, p.words + half * half_words(d), sh);
    else {
      empty_half(p, half);
      if (blockIdx.x == 0 && threadIdx.x == CT + 64) {
        p.ctl[3 + half] = (uint32_t)p.G;
        p.ctl[5 + (half ^ 1u)] = 0u;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int lane = threadIdx.x & 31;
    if (p.L > 0) {                  // this warp's first attention item and the cache rows of its first keys
      const int lgw = sh->lgw, W = 1 << lgw, ST = W * 8;
      const int item = (int)blockIdx.x * (NW >> lgw) + (warp >> lgw), kg = (warp & (W - 1)) * 8 + (lane >> 2);
      if (item < p.G * p.H) {
        const int pos = p.pos[item / p.H], slot = p.slot[item / p.H];
        auto row_at = [&](int j) {
          const int jb = p.block_of(j);
          return p.btab[(size_t)slot * p.max_lb + jb] * p.bs + (j - jb * p.bs);
        };
        const bool good = pos >= 0 && slot >= 0 && pos < p.max_ctx && p.block_of(pos) < p.max_lb;
        if (lane == 0) { sh->item_pos[warp] = pos; sh->item_slot[warp] = slot; sh->pos_row[warp] = good ? row_at(pos) : 0; }
        const int i = lane & 3;
        if (good && i < NB && kg + i * ST < pos) sh->item_row[warp][lane >> 2][i] = row_at(kg + i * ST);
      }
      __syncwarp();
    }
    // lane i < 12 holds the i-th pointer of this layer's record and of the next one's
    auto record = [&](int l) { return lane < 12 && l < p.L ? __ldg(reinterpret_cast<const unsigned long long*>(p.layers + l) + lane) : 0ull; };
    unsigned long long rec = record(0), nrec = record(1);
    auto ptr = [&](unsigned long long r, int i) { return reinterpret_cast<const bf16*>(__shfl_sync(0xffffffffu, r, i)); };
    int flip = 0;
    const uint32_t block = (uint32_t)slot_words(p.d);
    uint32_t *cur = p.words + (sh->launch & 1u) * half_words(p.d), *nxt = cur + block, *nx2 = nxt + block, *prv = nx2 + block;
#pragma unroll 1
    for (int k = 0; k < 4 * p.L + (p.head_w ? 1 : 0); k++) {
      const int l = k >> 2, j = k & 3, d = fresh(p.d);
      const uint32_t row = (uint32_t)MAX_ROWS * (d / 2);    // words: x at 0, mid at row, att at 2 row, qkv at 3 row, act at 6 row
      const bool head = k == 4 * p.L, ln = (j & 1) == 0;
      if (j == 0 && !head) wait_cleared(l, sh, p.wait_ns);
      if (j == 1) attention_phase<MT, HD, NB>(p, l, 5 * l + 1, cur + 3 * row, cur + 2 * row, satt, sh);
      Lin L;
      L.bias = ptr(rec, j == 0 ? 3 : j == 1 ? 5 : j == 2 ? 9 : 11);
      L.K = j == 3 ? 4 * d : d;
      L.N = j == 0 ? 3 * d : j == 2 ? 4 * d : d;
      L.kind = j == 0 ? PA : j == 1 ? PC : j == 2 ? PD : PE;
      L.seq = 5 * l + (j == 0 ? 0 : j + 1);
      L.src = j == 0 ? (l ? prv : nullptr) : cur + (j == 1 ? 2 : j == 2 ? 1 : 6) * row;
      L.res = j == 1 ? (l ? prv : nullptr) : j == 3 ? cur + row : nullptr;
      L.dst = cur + (j == 0 ? 3 : j == 1 ? 1 : j == 2 ? 6 : 0) * row;
      if (head) { L.bias = nullptr; L.N = p.V; L.kind = PH; L.dst = nullptr; }
      product<MT, LEFT>(p, L, ln, head ? p.n_rows : p.G, j == 3 && l + 1 == p.L, xs, red, flip, ring, sh);
      if (j == 3) {
        uint32_t* t = prv;
        prv = cur; cur = nxt; nxt = nx2; nx2 = t;
        rec = nrec;                    // (layer l + 2 is requested two layers ahead of its first use)
        nrec = record(l + 2);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sh->abort_flag) atomicCAS(p.err, 0, 9);
    const uint32_t launch = sh->launch;
    __threadfence();
    if (atomicAdd(p.ctl + 2, 1u) == gridDim.x - 1) {
      p.ctl[2] = 0;
      __threadfence();
      *reinterpret_cast<volatile uint32_t*>(p.ctl) = launch + 1u;
    }
  }
}

constexpr int fixed_bytes(int MT, int d) {         // shared memory beside the ring
  return 16 * MT * (d + PAD) + n_ln(d) * 4 * d + n_red(MT) * NW * LN_GROUPS * 64 * MT * 4 + NW * ATT_PITCH * 4 + (int)sizeof(Shared);
}
constexpr int ring_slots(int MT, int d) {
  const int n = (SMEM_LIMIT - fixed_bytes(MT, d)) / SLOT;
  return n < MAX_SLOTS ? n : MAX_SLOTS;
}
// Row groups of eight that one launch takes: by the shared memory that the normalised rows of wide models need beside a ring of at least the
// four chunks of a turn.
constexpr int max_mt(int d) { return d <= 1536 ? 4 : (d <= 3328 ? 2 : 1); }
static_assert(ring_slots(4, 1024) >= 4 && ring_slots(4, 1536) >= 4 && ring_slots(2, 3328) >= 4 && ring_slots(1, 4096) >= 4, "a turn's chunks fit");

template <int MT, int HD, int NB, int LEFT>
int launch(DecodeParams& p, int grid, cudaStream_t st) {
  p.slots = ring_slots(MT, p.d);
  const int smem = p.slots * SLOT + fixed_bytes(MT, p.d);
  p.lgw = 3;                                    // as many warps per (sequence, head) as keep all items in one turn
  while (p.lgw > 0 && (long)p.G * p.H << p.lgw > (long)grid * NW) p.lgw--;
  cudaError_t e = cudaFuncSetAttribute(decode_layers_k<MT, HD, NB, LEFT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { kh_set_error("decode_layers: shared memory opt-in failed: %s", cudaGetErrorString(e)); return -1; }
  // cooperative launch: the driver guarantees that all CTAs are resident together (or refuses the launch)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, decode_layers_k<MT, HD, NB, LEFT>, p);
  if (e != cudaSuccess) { kh_set_error("decode_layers launch failed: %s", cudaGetErrorString(e)); return -1; }
  return 0;
}
template <int HD, int LEFT>
int launch_rows(DecodeParams& p, int rows, int grid, cudaStream_t st) {
  if constexpr (HD == 32) {
    if (rows <= 16 && p.max_ctx > LONG_CTX) return rows <= 8 ? launch<1, HD, 4, LEFT>(p, grid, st) : launch<2, HD, 4, LEFT>(p, grid, st);
  }
  if (rows <= 8) return launch<1, HD, 2, LEFT>(p, grid, st);
  if (rows <= 16) return launch<2, HD, 2, LEFT>(p, grid, st);
  return launch<4, HD, HD == 32 ? 4 : 2, LEFT>(p, grid, st);
}
template <int HD>
int launch_width(DecodeParams& p, int rows, int grid, cudaStream_t st) {
  if (p.d % 1024 == 0) return launch_rows<HD, 4>(p, rows, grid, st);
  if (p.d < 1024) return p.d == 256 ? launch_rows<HD, 1>(p, rows, grid, st) : p.d == 512 ? launch_rows<HD, 2>(p, rows, grid, st) : launch_rows<HD, 3>(p, rows, grid, st);
  return launch_rows<HD, 0>(p, rows, grid, st);
}
int launch_any(DecodeParams& p, int hd, int rows, int grid, cudaStream_t st) {
  if (hd == 128) return launch_width<128>(p, rows, grid, st);
  if (hd == 64) return launch_width<64>(p, rows, grid, st);
  return launch_width<32>(p, rows, grid, st);
}

}  // namespace

// The decode batch sizes and model shapes the persistent decode kernel accepts.
extern "C" int kh_decode_layers_ok(int G, int d, int H, int hd, int max_ctx) {
  return G >= 1 && G <= MAX_ROWS && d >= 256 && d <= 4096 && d % 256 == 0 && H * hd == d && (hd == 32 || hd == 64 || hd == 128) &&
         max_ctx >= 1 && max_ctx <= 32768;
}

// Sequences of width d that one launch holds (more run in groups, and every group reads all weights again).
extern "C" int kh_decode_layers_rows(int d) { return 8 * max_mt(d); }

// Bytes of the workspace of activations (zero-initialised once, then only used by launches that follow one another).
extern "C" long kh_decode_layers_work_bytes(int d) { return CTL_BYTES + 2l * half_words(d) * 4; }

// x [G, d] holds the embedded tokens on entry and the last layer's output on return.  `layers`: device
// array of L records of twelve bf16 pointers (ln1_w, ln1_b, qkv_w, qkv_b, proj_w, proj_b, ln2_w, ln2_b,
// fc_w, fc_b, fcproj_w, fcproj_b).  With `head_w` ([V, d]) the kernel also writes
// logits[i, :V] = LNf(x[rows[i]]) head_w^T for i < n_rows (row pitch ld_logits).  `work`: the workspace,
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
  p.d = d; p.H = H; p.bs = bs; p.max_lb = max_lb; p.max_ctx = max_ctx;
  p.layers = (const LayerW*)layers;
  p.kc = (bf16*)kc; p.vc = (bf16*)vc; p.layer_elems = (size_t)layer_elems;
  p.btab = (const int*)btab;
  p.ctl = (uint32_t*)work;
  p.words = (uint32_t*)((uint8_t*)work + CTL_BYTES);
  p.inv_d = 1.f / (float)d;
  p.h_mul = (uint32_t)(((1ull << 32) + H - 1) / H);
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
    if (launch_any(p, hd, head_w && together && n_rows > n ? n_rows : n, grid, st)) return -1;
  }
  if (head_w && !together) {
    for (int r0 = 0; r0 < n_rows; r0 += cap) {
      const int n = n_rows - r0 < cap ? n_rows - r0 : cap;
      p.G = n; p.L = 0; p.x = (bf16*)x;
      set_head(r0, n);
      if (launch_any(p, hd, n, grid, st)) return -1;
    }
  }
  return 0;
}
