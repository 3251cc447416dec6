// bf16 GEMM family on the 5th-generation tensor cores (sm_100a).
//
//   C[M,N] (+)= op(A) * op(B)          fp32 accumulation in TMEM
//
// A is either K-major ([M,K] row-major) or M-major ([K,M] row-major); B is either K-major
// ([N,K] row-major, i.e. an nn.Linear weight) or N-major ([K,N] row-major).  That covers
// the three products of a linear layer without any transposed copies:
//   forward        Y  = X  * W^T      A K-major,  B K-major     (reference mm_nt_bf16o, kernels.cu:34-39)
//   input grad     dX = dY * W        A K-major,  B N-major     (reference mm_nn_bf16o, kernels.cu:55-60)
//   weight grad    dW = dY^T * X      A M-major,  B N-major     (reference mm_tn_bf16[_acc], kernels.cu:41-53)
//
// Structure: persistent CTAs (one per SM), 6 or 10 warps.  Warp 0 streams operand tiles with TMA
// into a ring of 128-byte-swizzled shared-memory stages; one lane of warp 1 issues
// tcgen05.mma (128 x BN x 16 per instruction) into one of two TMEM accumulator buffers and
// commits stage-release / accumulator-ready mbarriers; warps 2-9 (2-5 beyond K = 1024 and with
// column sums) drain the other accumulator with tcgen05.ld and run the fused epilogue, so the epilogue of tile i
// overlaps the main loop of tile i+1.
//
// Fused epilogues replace the reference's separate elementwise kernels
// (add_bias_k kernels.cu:174, bias_gelu_k :292, bias_residual_k :274, gelu_bwd_k :431,
// add_k :262) and the beta=1 weight-gradient accumulation.
//
// Bias gradients: with `colsum` set (weight-gradient products, A = dY in M-major form) four of the
// epilogue warps add up the columns of the A tiles while they sit in shared memory and the CTAs that own
// the first column of output tiles add the sums into colsum[M] -- the reference's separate
// colsum_k pass over dY (kernels.cu:511-524) disappears.  A stage is handed back to the TMA
// producer only after both the MMAs and these warps are done with it.
//
// Every mbarrier wait is bounded: on expiry the CTA stores a code in the library error word,
// all roles unwind, TMEM is released and the kernel returns.
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <string>
#include <unordered_map>

#include "common.cuh"

__device__ int g_kh_error_word = 0;
int* kh_error_word_dev() {
  static int* ptr[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  if (!ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_kh_error_word) == cudaSuccess) ptr[dev] = (int*)p;
  }
  return ptr[dev];
}

// ------------------------------------------------------------------------------- host util
static unsigned long long g_peer_wait_ns = 0;
unsigned long long kh_peer_wait_limit_ns() {
  if (g_peer_wait_ns == 0) {
    unsigned long long ms = 30000;
    if (const char* e = getenv("KHARON_PEER_WAIT_MS")) {
      const long v = atol(e);
      if (v > 0) ms = (unsigned long long)v;
    }
    g_peer_wait_ns = ms * 1000000ull;
  }
  return g_peer_wait_ns;
}
// Limit of every in-kernel wait on another rank, in milliseconds; returns the previous value.
extern "C" long kh_set_peer_wait_limit_ms(long ms) {
  const long old = (long)(kh_peer_wait_limit_ns() / 1000000ull);
  if (ms > 0) g_peer_wait_ns = (unsigned long long)ms * 1000000ull;
  return old;
}
static int g_pdl = -1;
int kh_pdl_enabled() {
  if (g_pdl < 0) {
    const char* e = getenv("KHARON_PDL");
    g_pdl = (e && e[0] == '0') ? 0 : 1;
  }
  return g_pdl;
}
// Programmatic dependent launch for all kernels of the library on/off; returns the previous setting.
extern "C" int kh_set_pdl(int on) {
  const int old = kh_pdl_enabled();
  g_pdl = on ? 1 : 0;
  return old;
}
static thread_local std::string g_host_err;
void kh_set_error(const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_host_err = buf;
}
extern "C" const char* kh_cuda_last_error() { return g_host_err.c_str(); }
extern "C" int kh_cuda_error_word(int reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_kh_error_word, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v != 0) {
    int z = 0;
    cudaMemcpyToSymbol(g_kh_error_word, &z, sizeof(int));
  }
  return v;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

struct TmapKey {
  uint64_t base, rows, cols, ld;
  uint32_t br, bc;
  bool operator==(const TmapKey& o) const { return memcmp(this, &o, sizeof(TmapKey)) == 0; }
};
struct TmapHash {
  size_t operator()(const TmapKey& k) const {
    uint64_t h = k.base * 0x9E3779B97F4A7C15ull;
    h ^= (k.rows + 0x632BE59BD9B4E019ull) + (h << 6) + (h >> 2);
    h ^= (k.cols * 31 + k.ld) + (h << 6) + (h >> 2);
    h ^= ((uint64_t)k.br << 32 | k.bc) + (h << 6) + (h >> 2);
    return (size_t)h;
  }
};
static size_t g_tmap_limit = 1u << 16;
// Test hook: number of cached descriptors after which the index is dropped (returns the old limit).
extern "C" long kh_tmap_cache_limit(long n) {
  const long old = (long)g_tmap_limit;
  if (n > 0) g_tmap_limit = (size_t)n;
  return old;
}

// Returns a descriptor that stays valid for the life of the process: callers hold the pointer
// across further look-ups (a launch fetches the A, B and output maps one after the other).
const CUtensorMap* kh_tmap_2d_bf16(const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                                   uint32_t box_rows, uint32_t box_cols) {
  static std::unordered_map<TmapKey, CUtensorMap*, TmapHash> cache;
  static std::mutex mu;
  TmapKey key;
  memset(&key, 0, sizeof(key));
  key.base = (uint64_t)base; key.rows = rows; key.cols = cols; key.ld = ld; key.br = box_rows; key.bc = box_cols;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  EncodeTiledFn fn = encode_fn();
  if (!fn) { kh_set_error("cuTensorMapEncodeTiled is not available from the driver"); return nullptr; }
  if (((uint64_t)base & 15) || ((ld * 2) & 15)) {
    kh_set_error("TMA operand needs a 16-byte aligned base and row pitch (base %p, ld %llu elements)", base,
                 (unsigned long long)ld);
    return nullptr;
  }
  CUtensorMap* m = new CUtensorMap;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult rc = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    delete m;
    kh_set_error("cuTensorMapEncodeTiled failed with %d (rows %llu cols %llu ld %llu box %ux%u)", (int)rc,
                 (unsigned long long)rows, (unsigned long long)cols, (unsigned long long)ld, box_rows, box_cols);
    return nullptr;
  }
  if (cache.size() >= g_tmap_limit) {
    // Buffers come from long-lived arenas, so this only bounds pathological churn.  The index is
    // dropped but the descriptors themselves are deliberately NOT freed (128 bytes each): pointers
    // handed out earlier, possibly a moment ago to the caller that triggered this insertion, must
    // not dangle.
    cache.clear();
  }
  cache[key] = m;
  return m;
}

const CUtensorMap* kh_tmap_3d_bf16(const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t ld1, uint64_t ld2,
                                   uint32_t box_d1, uint32_t box_d0) {
  struct Key3 {
    uint64_t v[6];
    uint32_t b[2];
    bool operator==(const Key3& o) const { return memcmp(this, &o, sizeof(Key3)) == 0; }
  };
  struct Hash3 {
    size_t operator()(const Key3& k) const {
      uint64_t h = 0x9E3779B97F4A7C15ull;
      for (int i = 0; i < 6; i++) h ^= (k.v[i] + 0x632BE59BD9B4E019ull) + (h << 6) + (h >> 2);
      h ^= ((uint64_t)k.b[0] << 32 | k.b[1]) + (h << 6) + (h >> 2);
      return (size_t)h;
    }
  };
  static std::unordered_map<Key3, CUtensorMap*, Hash3> cache;
  static std::mutex mu;
  Key3 key;
  memset(&key, 0, sizeof(key));
  key.v[0] = (uint64_t)base; key.v[1] = d0; key.v[2] = d1; key.v[3] = d2; key.v[4] = ld1; key.v[5] = ld2;
  key.b[0] = box_d1; key.b[1] = box_d0;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  EncodeTiledFn fn = encode_fn();
  if (!fn) { kh_set_error("cuTensorMapEncodeTiled is not available from the driver"); return nullptr; }
  if (((uint64_t)base & 15) || ((ld1 * 2) & 15) || ((ld2 * 2) & 15)) {
    kh_set_error("TMA operand needs a 16-byte aligned base and pitches (base %p, pitches %llu / %llu elements)", base,
                 (unsigned long long)ld1, (unsigned long long)ld2);
    return nullptr;
  }
  CUtensorMap* m = new CUtensorMap;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {ld1 * 2, ld2 * 2};
  cuuint32_t box[3] = {box_d0, box_d1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult rc = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    delete m;
    kh_set_error("cuTensorMapEncodeTiled (3-D) failed with %d", (int)rc);
    return nullptr;
  }
  if (cache.size() >= g_tmap_limit) cache.clear();      // descriptors stay allocated, see kh_tmap_2d_bf16
  cache[key] = m;
  return m;
}

// ------------------------------------------------------------------------------- kernel
enum { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2, EPI_BIAS_RESID = 3, EPI_DGELU = 4, EPI_RESID = 5, EPI_GELU = 6 };

struct GemmParams {
  int M, N, K;
  int a_mn, b_mn;          // operand majors (0 = K-major, 1 = M/N-major)
  void* C; int ldc;        // output, bf16 or fp32
  int out_fp32, accumulate;
  int epi;
  const bf16* bias;        // [N]
  bf16* aux; int ldaux;    // EPI_BIAS_GELU: pre-activation out (EPI_GELU: the same without it); EPI_BIAS_RESID/EPI_RESID: residual in; EPI_DGELU: pre-activation in
  float alpha;             // scales the accumulator before the epilogue
  float* colsum;           // [M] fp32 or null: colsum[m] (+)= sum_k op(A)[m, k]  (needs a_mn)
  int* err;                // library error word
};

// ---- epilogue arithmetic on pairs of columns (f32x2 of common.cuh): gelu_tanh and its derivative (common.cuh) with u = x (k + k c x^2)
__device__ __forceinline__ f32x2 gelu_tanh2(f32x2 x) {
  constexpr float k = 0.79788456f, c = 0.044715f;
  const f32x2 u = mul2(x, fma2(mul2(x, x), mk2(k * c, k * c), mk2(k, k))), h = mul2(x, mk2(0.5f, 0.5f));
  return fma2(h, mk2(tanhf(lo2(u)), tanhf(hi2(u))), h);
}
__device__ __forceinline__ f32x2 gelu_tanh_grad2(f32x2 x) {
  constexpr float k = 0.79788456f, c = 0.044715f;
  const f32x2 x2 = mul2(x, x), u = mul2(x, fma2(x2, mk2(k * c, k * c), mk2(k, k))), half = mk2(0.5f, 0.5f);
  const f32x2 t = mk2(tanhf(lo2(u)), tanhf(hi2(u)));
  const f32x2 s = fma2(mul2(t, mk2(-1.f, -1.f)), t, mk2(1.f, 1.f));                      // 1 - t^2
  return fma2(mul2(x, s), fma2(x2, mk2(1.5f * k * c, 1.5f * k * c), mk2(0.5f * k, 0.5f * k)), fma2(t, half, half));
}

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int GEMM_THREADS = 320;          // TMA, MMA and eight epilogue warps (or four and four column-sum warps); 192: four epilogue warps

// Staging buffer of an epilogue warp: 32 rows of 64 bytes (32 bf16 columns), the 16-byte pieces of a row exchanged by its index (conflict-free
// accesses both by row and by piece).
constexpr int EPI_BYTES = 32 * 64;

// PAIR: two CTAs of a cluster form one 256 x BN tile (tcgen05 cta_group::2).  Each CTA stages its
// own 128 rows of A and its own half of B, so a pair moves and re-reads 2/3 of the shared-memory
// bytes of two independent 128 x BN tiles.
template <int BN, bool PAIR = false> struct GemmCfg {
  static constexpr int BN_CTA = PAIR ? BN / 2 : BN;          // B rows (or columns) staged by one CTA
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN_CTA * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = PAIR ? 6 : ((BN == 256) ? 4 : (BN == 128 ? 6 : 8));
  static constexpr int TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/ + 8 * EPI_BYTES;
};

template <int BN, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p) {
  using Cfg = GemmCfg<BN, PAIR>;
  constexpr int TM = PAIR ? 2 * BM : BM;                       // rows of one scheduled tile
  const uint32_t crank = PAIR ? cluster_ctarank() : 0u;        // 0 = leader (issues the MMAs)
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int n_workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_al + Cfg::STAGES * Cfg::STAGE_BYTES);
  // bars: full[STAGES], empty[STAGES], tfull[2], tempty[2], free[STAGES], then tmem base word + abort flag
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = bar_full + 8 * Cfg::STAGES;
  const uint32_t bar_tfull = bar_empty + 8 * Cfg::STAGES;
  const uint32_t bar_tempty = bar_tfull + 16;
  const uint32_t bar_free = bar_tempty + 16;         // column-sum warps are done with the stage
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * Cfg::STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const bool csum = p.colsum != nullptr;
  const int parts = !csum && blockDim.x == GEMM_THREADS ? 2 : 1;      // epilogue warps to a TMEM quadrant

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (p.M + TM - 1) / TM, tiles_n = (p.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; s++) {
      mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); mbar_init(bar_free + 8 * s, 4);
    }
    // accumulator-free barrier: one arrival per epilogue warp of every CTA that reads the accumulator
    for (int a = 0; a < 2; a++) { mbar_init(bar_tfull + 8 * a, 1); mbar_init(bar_tempty + 8 * a, (PAIR ? 2 : 1) * 4 * parts); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(smem_u32(tmem_slot), Cfg::TMEM_COLS); tmem_relinquish_pair(); }
    else { tmem_alloc(smem_u32(tmem_slot), Cfg::TMEM_COLS); tmem_relinquish(); }
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tma_a); tma_prefetch_desc(&tma_b); }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the peer's barriers are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                        // operands and outputs belong to earlier kernels of the stream up to here
  pdl_launch_dependents();

  // tile id -> (tm, tn): bands of 8 M-tiles, N fastest inside a band keeps both panels in L2
  auto tile_coord = [&](int t, int& tm, int& tn) {
    const int GROUP = 8;
    int band = t / (GROUP * tiles_n);
    int first = band * GROUP;
    int gsz = min(GROUP, tiles_m - first);
    int r = t - band * GROUP * tiles_n;
    tm = first + r % gsz;
    tn = r / gsz;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int it = 0;
      bool ok = true;
      for (int t = worker; ok && t < num_tiles; t += n_workers) {
        int tm, tn;
        tile_coord(t, tm, tn);
        const int m0 = tm * TM + (int)crank * BM;               // first A row of this CTA
        const int n0 = tn * BN + (int)crank * Cfg::BN_CTA;      // first B row/column of this CTA
        for (int kb = 0; kb < num_kb; kb++, it++) {
          const int s = it % Cfg::STAGES;
          const uint32_t ph = (it / Cfg::STAGES) & 1;
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, 2, p.err)) { ok = false; break; }
          if (csum && !mbar_wait(bar_free + 8 * s, ph ^ 1, abort_flag, 2, p.err)) { ok = false; break; }
          const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
          if (!PAIR) {
            mbar_expect_tx(bar_full + 8 * s, Cfg::STAGE_BYTES);
            if (!p.a_mn) tma_load_2d(sa, &tma_a, bar_full + 8 * s, kb * BK, m0);
            else
              for (int j = 0; j < BM / 64; j++) tma_load_2d(sa + j * (BK * 128), &tma_a, bar_full + 8 * s, m0 + j * 64, kb * BK);
            if (!p.b_mn) tma_load_2d(sb, &tma_b, bar_full + 8 * s, kb * BK, n0);
            else
              for (int j = 0; j < BN / 64; j++) tma_load_2d(sb + j * (BK * 128), &tma_b, bar_full + 8 * s, n0 + j * 64, kb * BK);
          } else {
            // both CTAs credit the leader's barrier; the leader expects the bytes of the whole pair
            const uint32_t lbar = mapa_shared(bar_full + 8 * s, 0);
            if (crank == 0) mbar_expect_tx(bar_full + 8 * s, 2 * Cfg::STAGE_BYTES);
            if (!p.a_mn) tma_load_2d_pair(sa, &tma_a, lbar, kb * BK, m0);
            else
              for (int j = 0; j < BM / 64; j++) tma_load_2d_pair(sa + j * (BK * 128), &tma_a, lbar, m0 + j * 64, kb * BK);
            if (!p.b_mn) tma_load_2d_pair(sb, &tma_b, lbar, kb * BK, n0);
            else
              for (int j = 0; j < Cfg::BN_CTA / 64; j++) tma_load_2d_pair(sb + j * (BK * 128), &tma_b, lbar, n0 + j * 64, kb * BK);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (crank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(TM, BN, p.a_mn, p.b_mn);
      // K-major: LBO unused (encoded 16 B), SBO 1024; MN-major: LBO = one 64-wide slab (BK rows x 128 B), SBO 1024
      const uint32_t a_lbo = p.a_mn ? BK * 128 : 16, b_lbo = p.b_mn ? BK * 128 : 16;
      const uint32_t a_kstep = p.a_mn ? (UMMA_K * 128) >> 4 : (UMMA_K * 2) >> 4;
      const uint32_t b_kstep = p.b_mn ? (UMMA_K * 128) >> 4 : (UMMA_K * 2) >> 4;
      int it = 0, tcount = 0;
      bool ok = true;
      for (int t = worker; ok && t < num_tiles; t += n_workers, tcount++) {
        const int acc = tcount & 1;
        const uint32_t aph = (tcount >> 1) & 1;
        if (!mbar_wait(bar_tempty + 8 * acc, aph ^ 1, abort_flag, 4, p.err)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; kb++, it++) {
          const int s = it % Cfg::STAGES;
          const uint32_t ph = (it / Cfg::STAGES) & 1;
          if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, 1, p.err)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
          uint64_t adesc = umma_desc_sw128(sa, a_lbo, 1024);
          uint64_t bdesc = umma_desc_sw128(sb, b_lbo, 1024);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; k++) {
            if (PAIR) umma_f16_ss_pair(d_tmem, adesc + (uint64_t)(k * a_kstep), bdesc + (uint64_t)(k * b_kstep), idesc,
                                       (kb > 0 || k > 0) ? 1u : 0u);
            else umma_f16_ss(d_tmem, adesc + (uint64_t)(k * a_kstep), bdesc + (uint64_t)(k * b_kstep), idesc,
                             (kb > 0 || k > 0) ? 1u : 0u);
          }
          // stage reusable (in both CTAs of a pair) once these MMAs retire
          if (PAIR) umma_commit_pair(bar_empty + 8 * s, 3); else umma_commit(bar_empty + 8 * s);
        }
        if (ok) { if (PAIR) umma_commit_pair(bar_tfull + 8 * acc, 3); else umma_commit(bar_tfull + 8 * acc); }
      }
    }
  } else if (csum && warp >= 6) {
    // ------------------------------------------------------------------ column sums of A (bias gradient)
    // Present only in launches with column sums.  A stage is read after the MMAs that consume it
    // have retired (its "empty" barrier, which also reaches the second CTA of a pair) and before the
    // producer may refill it (the "free" barrier).  Warp cw owns columns [32 cw, 32 cw + 32) of the
    // 128-column A tile: four 16-byte chunks of one 64-column slab.  Lane = 8 p + 4 h + c4 reads
    // chunk c4 of rows 8 i + p + 4 h (i = 0..7): the two rows of a quarter-warp differ in bit 2, so
    // the 128-byte swizzle puts them in different bank halves.  The warp needs no other warp's
    // data, so there is no barrier between the four.
    const int cw = warp - 6;
    const int c4 = lane & 3, rsel = ((lane >> 3) & 3) + 4 * ((lane >> 2) & 1);
    const uint32_t slab_off = (uint32_t)(cw >> 1) * (BK * 128);
    const int chunk = (cw & 1) * 4 + c4;
    int it = 0;
    bool ok = true;
    for (int t = worker; ok && t < num_tiles; t += n_workers) {
      int tm, tn;
      tile_coord(t, tm, tn);
      const bool mine = (tn == 0);
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; j++) acc[j] = 0.f;
      for (int kb = 0; kb < num_kb; kb++, it++) {
        const int s = it % Cfg::STAGES;
        const uint32_t ph = (it / Cfg::STAGES) & 1;
        if (!mbar_wait(bar_empty + 8 * s, ph, abort_flag, 2, p.err)) { ok = false; break; }
        if (mine) {
          const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES + slab_off;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int r = 8 * i + rsel;
            uint4 v;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                         : "r"(sa + (uint32_t)r * 128u + (uint32_t)((chunk ^ (r & 7)) << 4)));
            float2 f0 = unpack_bf16(v.x), f1 = unpack_bf16(v.y), f2 = unpack_bf16(v.z), f3 = unpack_bf16(v.w);
            acc[0] += f0.x; acc[1] += f0.y; acc[2] += f1.x; acc[3] += f1.y;
            acc[4] += f2.x; acc[5] += f2.y; acc[6] += f3.x; acc[7] += f3.y;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_free + 8 * s);
      }
      if (ok && mine) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 4);
          acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 8);
          acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
        }
        if (lane < 4) {
          const int m0 = tm * TM + (int)crank * BM + cw * 32 + c4 * 8;
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (m0 + j < p.M) p.colsum[m0 + j] = p.accumulate ? p.colsum[m0 + j] + acc[j] : acc[j];
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    // Four warps with all columns of a tile, or eight, two per TMEM quadrant, with every second 32 columns each (see gemm_threads): the two
    // halves of a line are then written at about the same time.  With half of the tile's columns each, 8192 x 2048 x 512 took 18.2 us plain, 23.7 with
    // GELU and 27.3 with its pre-activation too, 28.4 times GELU'; so 17.4, 21.7, 25.3, 26.7; 8192 x 1536 x 512 15.3 and 14.6.  (Sixteen warps: 20.3
    // plain; steps of 64 columns in whole lines 17.6, but 29 with GELU and pre-activation: fewer steps overlap.)
    const int q = warp & 3;                    // TMEM lane quadrant this warp may access
    const int part = (warp - 2) >> 2, step = 32 * parts;
    // A thread owns a row of the accumulator, but global memory is read and written in pieces of 16 bytes, four neighbouring
    // lanes to a row of the 32-column chunk: the warp turns the chunk around in its staging buffer.  With every lane on its own row an
    // access touched 32 lines, and the load / store unit bounded the products of narrow models (9216 x 1536 x 512:
    // 23.6 us plain, 30 with a residual, 38 with GELU and its pre-activation; cuBLAS plain 14.1).
    const uint32_t stg = smem_base + Cfg::STAGES * Cfg::STAGE_BYTES + 256 + (warp - 2) * EPI_BYTES;
    const int prow = lane >> 2, pcol = (lane & 3) * 8;          // this lane's piece: row 8 j + prow, columns pcol ..
    auto staged = [&](int r, int piece) { return stg + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4); };
    auto put_row = [&](const uint32_t (&w)[16]) {                // own row, bf16 pairs -> staging
#pragma unroll
      for (int j = 0; j < 4; j++)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(staged(lane, j)), "r"(w[4 * j]), "r"(w[4 * j + 1]), "r"(w[4 * j + 2]),
                     "r"(w[4 * j + 3]) : "memory");
    };
    auto lds = [&](uint32_t a) {
      uint4 u;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(a) : "memory");
      return u;
    };
    auto store_rows = [&](bf16* base, int ld, int r0, int col, const uint32_t (&w)[16]) {      // 32 rows from r0, columns col ..
      put_row(w);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint4 u = lds(staged(j * 8 + prow, lane & 3));
        if (r0 + j * 8 + prow < p.M) *reinterpret_cast<uint4*>(base + (size_t)(r0 + j * 8 + prow) * ld + col + pcol) = u;
      }
      __syncwarp();
    };
    int tcount = 0;
    bool ok = true;
    for (int t = worker; ok && t < num_tiles; t += n_workers, tcount++) {
      int tm, tn;
      tile_coord(t, tm, tn);
      const int acc = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1;
      const int row0 = tm * TM + (int)crank * BM + q * 32, row = row0 + lane;
      const bool row_ok = row < p.M;
      const bool use_bias = (p.epi == EPI_BIAS || p.epi == EPI_BIAS_GELU || p.epi == EPI_BIAS_RESID || p.epi == EPI_GELU);
      const bool use_aux = (p.epi == EPI_BIAS_RESID || p.epi == EPI_RESID || p.epi == EPI_DGELU);
      // Operands of the epilogue are fetched one 32-column chunk ahead (the first chunk before the
      // accumulator is even complete), so their DRAM latency is not paid once per chunk.
      uint4 nb[4] = {}, nx[4] = {};
      auto fetch = [&](int c0) {
        const int col = tn * BN + c0;
        if (c0 >= BN || col + 32 > p.N) return;
        if (use_bias) {
          const uint4* bp = reinterpret_cast<const uint4*>(p.bias + col);
#pragma unroll
          for (int j = 0; j < 4; j++) nb[j] = __ldg(bp + j);
        }
        if (use_aux) {
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (row0 + j * 8 + prow < p.M) nx[j] = *reinterpret_cast<const uint4*>(p.aux + (size_t)(row0 + j * 8 + prow) * p.ldaux + col + pcol);
        }
      };
      if (use_aux && row_ok) {
        const char* ap = reinterpret_cast<const char*>(p.aux + (size_t)row * p.ldaux + tn * BN);
        const int nbytes = min(BN, p.N - tn * BN) * 2;
        for (int b = 128 * (1 + part); b < nbytes; b += 128 * parts) prefetch_l2(ap + b);
      }
      fetch(32 * part);
      if (!mbar_wait(bar_tfull + 8 * acc, aph, abort_flag, 3, p.err)) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
#pragma unroll 1
      for (int c0 = 32 * part; c0 < BN; c0 += step) {
        const int col = tn * BN + c0;
        if (col >= p.N) break;                 // uniform across the warp
        uint32_t r[32];
        tmem_ld32(taddr + c0, r);
        tmem_ld_wait();
        if (col + 32 <= p.N) {                 // uniform over the warp: rows past the end take part without memory accesses
          // With K of a few hundred this arithmetic and the stores bound a tile, not its MMAs: columns in pairs, and one rounding to bf16 for the
          // stored pre-activation and the argument of its GELU (8192 x 2048 x 512: GELU with pre-activation 31.4 us column by column, 27.4 so; times
          // GELU' 34.3 and 28.8; then see the order of the steps above).
          f32x2 v[16];
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; i++) v[i] = mk2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          if (p.alpha != 1.f) {
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = mul2(v[i], mk2(p.alpha, p.alpha));
          }
          if (use_bias) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
              v[4 * j] = add2(v[4 * j], un2(nb[j].x)); v[4 * j + 1] = add2(v[4 * j + 1], un2(nb[j].y));
              v[4 * j + 2] = add2(v[4 * j + 2], un2(nb[j].z)); v[4 * j + 3] = add2(v[4 * j + 3], un2(nb[j].w));
            }
          }
          if (!use_aux) fetch(c0 + step);
          if (p.epi == EPI_BIAS_GELU || p.epi == EPI_GELU) {
            // the stored pre-activation is bf16; apply GELU to the rounded value so that the
            // backward pass (which only sees the bf16 copy) differentiates the same function
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = pack2(v[i]);
            // (without a backward pass nobody reads the pre-activation: 4200 x 4096 x 1024 34.3 us with its store, 29.2 without)
            if (p.epi == EPI_BIAS_GELU) store_rows(p.aux, p.ldaux, row0, col, w);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = gelu_tanh2(un2(w[i]));
          } else if (use_aux) {
#pragma unroll
            for (int j = 0; j < 4; j++)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(staged(j * 8 + prow, lane & 3)), "r"(nx[j].x), "r"(nx[j].y),
                           "r"(nx[j].z), "r"(nx[j].w) : "memory");
            fetch(c0 + step);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const uint4 b = lds(staged(lane, j));
              w[4 * j] = b.x; w[4 * j + 1] = b.y; w[4 * j + 2] = b.z; w[4 * j + 3] = b.w;
            }
            if (p.epi == EPI_DGELU) {
#pragma unroll
              for (int i = 0; i < 16; i++) v[i] = mul2(v[i], gelu_tanh_grad2(un2(w[i])));
            } else {
#pragma unroll
              for (int i = 0; i < 16; i++) v[i] = add2(v[i], un2(w[i]));
            }
            __syncwarp();
          }
          if (!p.out_fp32) {
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = pack2(v[i]);
            store_rows(reinterpret_cast<bf16*>(p.C), p.ldc, row0, col, w);
          } else if (row_ok) {
            float* cp = reinterpret_cast<float*>(p.C) + (size_t)row * p.ldc + col;
            if (p.accumulate) {
#pragma unroll
              for (int j = 0; j < 8; j++) red_add_v4_f32(cp + 4 * j, lo2(v[2 * j]), hi2(v[2 * j]), lo2(v[2 * j + 1]), hi2(v[2 * j + 1]));
            } else {
#pragma unroll
              for (int j = 0; j < 8; j++)
                reinterpret_cast<float4*>(cp)[j] = make_float4(lo2(v[2 * j]), hi2(v[2 * j]), lo2(v[2 * j + 1]), hi2(v[2 * j + 1]));
            }
          }
        } else if (row_ok) {                   // ragged last columns
          // Everything is read before anything is written: the compiler keeps a load behind the stores of the column before it (bias fetched column
          // by column / ahead: 455 x 920 x 512 with GELU and pre-activation 16.0 / 11.5 us, 125 x 5848 x 1208 with residual 18.6 / 12.9, 16020 x 144 x 80 times
          // GELU' 13.5 / 11.5).
          float* const cf = reinterpret_cast<float*>(p.C) + (size_t)row * p.ldc + col;
          bf16* const ap = p.aux + (size_t)row * p.ldaux + col;
          float v[32], a[32];
#pragma unroll
          for (int i = 0; i < 32; i++) {
            v[i] = __uint_as_float(r[i]) * p.alpha;
            a[i] = 0.f;
          }
          if (use_bias)
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (col + i < p.N) v[i] += __bfloat162float(p.bias[col + i]);
          if (use_aux)
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (col + i < p.N) a[i] = __bfloat162float(ap[i]);
          if (p.epi == EPI_BIAS_GELU || p.epi == EPI_GELU) {
#pragma unroll
            for (int i = 0; i < 32; i++) {
              const bf16 pre = __float2bfloat16(v[i]);
              if (p.epi == EPI_BIAS_GELU && col + i < p.N) ap[i] = pre;
              v[i] = gelu_tanh(__bfloat162float(pre));
            }
          } else if (use_aux) {
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = p.epi == EPI_DGELU ? v[i] * gelu_tanh_grad(a[i]) : v[i] + a[i];
          }
          if (!p.out_fp32) {
            bf16* const cp = reinterpret_cast<bf16*>(p.C) + (size_t)row * p.ldc + col;
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (col + i < p.N) cp[i] = __float2bfloat16(v[i]);
          } else {
            if (p.accumulate)
#pragma unroll
              for (int i = 0; i < 32; i++)
                if (col + i < p.N) a[i] = cf[i];
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (col + i < p.N) cf[i] = p.accumulate ? a[i] + v[i] : v[i];
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(mapa_shared(bar_tempty + 8 * acc, 0));   // the leader issues the MMAs
        else mbar_arrive(bar_tempty + 8 * acc);
      }
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // no CTA leaves while its peer may still signal its barriers
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS); else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------- split-K kernel
// Products whose output has too few tiles for the chip and whose K is long (weight gradients of narrow layers: K is the number
// of tokens; input gradients and forward products of few rows): a k-block costs a CTA 0.4-0.5 us whatever its tile width (the
// chain TMA -> tcgen05.mma -> release), so one CTA per tile takes K / 64 of them one after the other while most SMs idle.
// Here the 2, 4 or 8 CTAs of a cluster share one 128 x BN tile: CTA r multiplies the r-th slice of K, leaves its fp32
// partial tile in its own shared memory (the operand stages are free by then), and after a cluster barrier every CTA adds
// its 128 / split rows over the CTAs in rank order through distributed shared memory and runs the epilogue on them.  No
// workspace and no atomics; the order of the additions is fixed, so results are reproducible.
// PAIR: the 2, 3 or 4 members of the cluster are CTA pairs with a 256 x 256 tile (cta_group::2).  A k-block takes a pair as long as a
// CTA with its 128 x 128 tile (0.36 and 0.34 us, bound by the operands' way from L2) and covers four times the output.
// Measured (dW with column sums, one CTA per tile / CTAs share K / pairs share K, us, K = 9216): 512 x 512 49.1 / 18.2 / 20.2, 1536 x 512 49.7 / 30.9 / 21.8, 2048 x
// 512 50.2 / 31.6 / 27.3; K = 8192: 1024 x 1024 44.8 / 28.6 / 25.0; K = 4096: 1024 x 256 30.2 / 15.6, 2048 x 1024 26.7 / - / 21.8, 1536 x 512 25.0 / 18.1 /
// 15.0; forward 128 x 1024 x 4096: 27.9 / 13.8.
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
// Epilogue of four adjacent columns (col % 4 == 0) of one row; the arithmetic and rounding points of gemm_kernel.  Its operands are read by
// epilogue4_fetch, ahead of the sum (0 where there are none).
struct Epi4 { uint2 bias, aux; };
__device__ __forceinline__ uint2 load4(const bf16* a, int n) {
  if (n >= 4) return *reinterpret_cast<const uint2*>(a);
  uint32_t w[3] = {0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (i < n) w[i] = *reinterpret_cast<const uint16_t*>(a + i);
  return make_uint2(w[0] | w[1] << 16, w[2]);
}
__device__ __forceinline__ void epilogue4_fetch(const GemmParams& p, int row, int col, Epi4& e) {
  const int n = p.N - col;
  e.bias = e.aux = make_uint2(0u, 0u);
  if (p.epi == EPI_BIAS || p.epi == EPI_BIAS_GELU || p.epi == EPI_BIAS_RESID || p.epi == EPI_GELU) e.bias = load4(p.bias + col, n);
  if (p.epi == EPI_BIAS_RESID || p.epi == EPI_RESID || p.epi == EPI_DGELU) e.aux = load4(p.aux + (size_t)row * p.ldaux + col, n);
}
__device__ __forceinline__ void epilogue4(const GemmParams& p, int row, int col, float (&v)[4], const Epi4& e) {
  const int n = min(4, p.N - col);
  const float2 b0 = unpack_bf16(e.bias.x), b1 = unpack_bf16(e.bias.y);
  v[0] = v[0] * p.alpha + b0.x; v[1] = v[1] * p.alpha + b0.y; v[2] = v[2] * p.alpha + b1.x; v[3] = v[3] * p.alpha + b1.y;
  if (p.epi == EPI_BIAS_GELU || p.epi == EPI_GELU) {
    if (p.epi == EPI_BIAS_GELU) {
      bf16* ap = p.aux + (size_t)row * p.ldaux + col;
      if (n == 4) *reinterpret_cast<uint2*>(ap) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
      else for (int i = 0; i < n; i++) ap[i] = __float2bfloat16(v[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = gelu_tanh(__bfloat162float(__float2bfloat16(v[i])));
  } else if (p.epi == EPI_BIAS_RESID || p.epi == EPI_RESID || p.epi == EPI_DGELU) {
    const float2 a = unpack_bf16(e.aux.x), b = unpack_bf16(e.aux.y);
    const float x[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = p.epi == EPI_DGELU ? v[i] * gelu_tanh_grad(x[i]) : v[i] + x[i];
  }
  if (p.out_fp32) {
    float* cp = reinterpret_cast<float*>(p.C) + (size_t)row * p.ldc + col;
    if (n == 4) {
      if (p.accumulate) red_add_v4_f32(cp, v[0], v[1], v[2], v[3]);
      else *reinterpret_cast<float4*>(cp) = make_float4(v[0], v[1], v[2], v[3]);
    } else for (int i = 0; i < n; i++) cp[i] = p.accumulate ? cp[i] + v[i] : v[i];
  } else {
    bf16* cp = reinterpret_cast<bf16*>(p.C) + (size_t)row * p.ldc + col;
    if (n == 4) *reinterpret_cast<uint2*>(cp) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    else for (int i = 0; i < n; i++) cp[i] = __float2bfloat16(v[i]);
  }
}

template <int BN, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p,
                   int split) {
  using Cfg = GemmCfg<BN, PAIR>;
  constexpr int PITCH = BN + 4;                      // floats per row of the partial tile: conflict-free 16-byte rows
  static_assert((BM * PITCH + BM) * 4 <= Cfg::STAGES * Cfg::STAGE_BYTES, "the partial tile reuses the operand stages");
  const uint32_t ctarank = cluster_ctarank(), rank = PAIR ? ctarank >> 1 : ctarank;      // slice of K
  const uint32_t crank = PAIR ? ctarank & 1u : 0u, leader = ctarank & ~1u;                // half of the pair's tile
  constexpr int TM = PAIR ? 2 * BM : BM;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_al + Cfg::STAGES * Cfg::STAGE_BYTES);
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * Cfg::STAGES, bar_free = bar_empty + 8 * Cfg::STAGES,
                 bar_tfull = bar_free + 8 * Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * Cfg::STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const bool csum = p.colsum != nullptr;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_m = (p.M + TM - 1) / TM, tile = (int)blockIdx.x / (PAIR ? 2 * split : split);
  const int m0 = (tile % tiles_m) * TM + (int)crank * BM, tn = tile / tiles_m, n0 = tn * BN, nb0 = n0 + (int)crank * Cfg::BN_CTA;
  const int num_kb = (p.K + BK - 1) / BK, per = (num_kb + split - 1) / split;
  const int kb0 = min(num_kb, (int)rank * per), nkb = min(num_kb, kb0 + per) - kb0;       // the launcher leaves no slice empty

  if (tid == 0) {
    for (int s = 0; s < Cfg::STAGES; s++) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); mbar_init(bar_free + 8 * s, 4); }
    mbar_init(bar_tfull, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(smem_u32(tmem_slot), BN); tmem_relinquish_pair(); }
    else { tmem_alloc(smem_u32(tmem_slot), BN); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the barriers of the pair are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();

  bool ok = true;
  float cs[8];
#pragma unroll
  for (int j = 0; j < 8; j++) cs[j] = 0.f;
  if (warp == 0) {
    if (elect_one()) {
      for (int i = 0; i < nkb; i++) {
        const int s = i % Cfg::STAGES, kb = kb0 + i;
        const uint32_t ph = (i / Cfg::STAGES) & 1;
        if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, 2, p.err)) break;
        if (csum && !mbar_wait(bar_free + 8 * s, ph ^ 1, abort_flag, 2, p.err)) break;
        const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
        if (PAIR) {
          // both CTAs credit the leader's barrier; the leader expects the bytes of the pair
          const uint32_t lbar = mapa_shared(bar_full + 8 * s, leader);
          if (crank == 0) mbar_expect_tx(bar_full + 8 * s, 2 * Cfg::STAGE_BYTES);
          if (!p.a_mn) tma_load_2d_pair(sa, &tma_a, lbar, kb * BK, m0);
          else
            for (int j = 0; j < BM / 64; j++) tma_load_2d_pair(sa + j * (BK * 128), &tma_a, lbar, m0 + j * 64, kb * BK);
          if (!p.b_mn) tma_load_2d_pair(sb, &tma_b, lbar, kb * BK, nb0);
          else
            for (int j = 0; j < Cfg::BN_CTA / 64; j++) tma_load_2d_pair(sb + j * (BK * 128), &tma_b, lbar, nb0 + j * 64, kb * BK);
        } else {
          mbar_expect_tx(bar_full + 8 * s, Cfg::STAGE_BYTES);
          if (!p.a_mn) tma_load_2d(sa, &tma_a, bar_full + 8 * s, kb * BK, m0);
          else
            for (int j = 0; j < BM / 64; j++) tma_load_2d(sa + j * (BK * 128), &tma_a, bar_full + 8 * s, m0 + j * 64, kb * BK);
          if (!p.b_mn) tma_load_2d(sb, &tma_b, bar_full + 8 * s, kb * BK, n0);
          else
            for (int j = 0; j < BN / 64; j++) tma_load_2d(sb + j * (BK * 128), &tma_b, bar_full + 8 * s, n0 + j * 64, kb * BK);
        }
      }
    }
  } else if (warp == 1) {
    if (crank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(TM, BN, p.a_mn, p.b_mn);
      const uint16_t mask = (uint16_t)(3u << leader);
      const uint32_t a_lbo = p.a_mn ? BK * 128 : 16, b_lbo = p.b_mn ? BK * 128 : 16;
      const uint32_t a_kstep = p.a_mn ? (UMMA_K * 128) >> 4 : (UMMA_K * 2) >> 4;
      const uint32_t b_kstep = p.b_mn ? (UMMA_K * 128) >> 4 : (UMMA_K * 2) >> 4;
      for (int i = 0; ok && i < nkb; i++) {
        const int s = i % Cfg::STAGES;
        if (!mbar_wait(bar_full + 8 * s, (i / Cfg::STAGES) & 1, abort_flag, 1, p.err)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
        const uint64_t adesc = umma_desc_sw128(sa, a_lbo, 1024), bdesc = umma_desc_sw128(sb, b_lbo, 1024);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; k++)
          if (PAIR) umma_f16_ss_pair(tmem, adesc + (uint64_t)(k * a_kstep), bdesc + (uint64_t)(k * b_kstep), idesc, (i > 0 || k > 0) ? 1u : 0u);
          else umma_f16_ss(tmem, adesc + (uint64_t)(k * a_kstep), bdesc + (uint64_t)(k * b_kstep), idesc, (i > 0 || k > 0) ? 1u : 0u);
        if (PAIR) umma_commit_pair(bar_empty + 8 * s, mask); else umma_commit(bar_empty + 8 * s);
      }
      if (ok) { if (PAIR) umma_commit_pair(bar_tfull, mask); else umma_commit(bar_tfull); }
    }
  } else if (csum && warp >= 6) {
    // column sums of this CTA's A tiles, see gemm_kernel
    const int cw = warp - 6;
    const int c4 = lane & 3, rsel = ((lane >> 3) & 3) + 4 * ((lane >> 2) & 1), chunk = (cw & 1) * 4 + c4;
    for (int i = 0; i < nkb; i++) {
      const int s = i % Cfg::STAGES;
      if (!mbar_wait(bar_empty + 8 * s, (i / Cfg::STAGES) & 1, abort_flag, 2, p.err)) break;
      if (tn == 0) {
        const uint32_t sa = smem_base + s * Cfg::STAGE_BYTES + (uint32_t)(cw >> 1) * (BK * 128);
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const int r = 8 * q + rsel;
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(sa + (uint32_t)r * 128u + (uint32_t)((chunk ^ (r & 7)) << 4)));
          const float2 f0 = unpack_bf16(v.x), f1 = unpack_bf16(v.y), f2 = unpack_bf16(v.z), f3 = unpack_bf16(v.w);
          cs[0] += f0.x; cs[1] += f0.y; cs[2] += f1.x; cs[3] += f1.y;
          cs[4] += f2.x; cs[5] += f2.y; cs[6] += f3.x; cs[7] += f3.y;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_free + 8 * s);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      cs[j] += __shfl_xor_sync(0xffffffffu, cs[j], 4);
      cs[j] += __shfl_xor_sync(0xffffffffu, cs[j], 8);
      cs[j] += __shfl_xor_sync(0xffffffffu, cs[j], 16);
    }
  }
  __syncwarp();
  if (warp >= 2 && warp < 6) mbar_wait(bar_tfull, 0, abort_flag, 3, p.err);
  tc_fence_after();
  __syncthreads();                   // every MMA has retired and the column-sum warps are done: the stages are free
  const uint32_t tile_smem = smem_base, csum_smem = smem_base + BM * PITCH * 4;
  tc_fence_after();
  if (warp >= 2) {                   // two warps to a TMEM quadrant, half of the columns each
    const int q = warp & 3, row = q * 32 + lane, half = warp >= 6 ? BN / 2 : 0;
#pragma unroll 1
    for (int c = half; c < half + BN / 2; c += 32) {
      uint32_t r[32];
      tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 8; j++)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile_smem + (uint32_t)(row * PITCH + c + 4 * j) * 4u),
                     "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3]) : "memory");
    }
  }
  if (csum && warp >= 6 && lane < 4) {
#pragma unroll
    for (int j = 0; j < 8; j++)
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(csum_smem + (uint32_t)((warp - 6) * 32 + lane * 8 + j) * 4u), "f"(cs[j]) : "memory");
  }
  tc_fence_before();
  // The tail is a chain of latencies: the reads of all partial tiles (and of the abort flags) go out together, the epilogue's operands before
  // the barrier (128 x 1024 x 4096 with bias and residual 9.2 us with one read after the other and four warps leaving the tile, 8.0 so;
  // 18 x 256 x 1024 6.3 and 5.2; dW 768 x 256 x 4096 10.1 and 9.2).
  const int first = (int)rank * BM / split, rows = ((int)rank + 1) * BM / split - first, items = rows * (BN / 4);
  auto place = [&](int i, int& r, int& c) {
    r = first + i / (BN / 4); c = (i % (BN / 4)) * 4;
    return i < items && m0 + r < p.M && n0 + c < p.N;
  };
  int r, c;
  Epi4 e;
  if (place(tid, r, c)) epilogue4_fetch(p, m0 + r, n0 + c, e);
  cluster_sync_all();
  const uint32_t bad = lane < (PAIR ? 2 * split : split) ? ld_cluster_u32(mapa_shared(smem_u32((const void*)abort_flag), lane)) : 0u;
  float4 f[8];
  auto partials = [&](int r, int c) {
    const uint32_t at = tile_smem + (uint32_t)(r * PITCH + c) * 4u;
#pragma unroll
    for (int s = 0; s < 8; s++)
      if (s < split) f[s] = ld_cluster_v4(mapa_shared(at, PAIR ? 2 * s + crank : s));
  };
  bool in = place(tid, r, c);
  if (in) partials(r, c);
  const bool all_ok = !__any_sync(0xffffffffu, bad != 0);
  if (all_ok) {
    for (int i = tid; i < items; i += GEMM_THREADS) {
      if (i != tid) {
        in = place(i, r, c);
        if (in) { epilogue4_fetch(p, m0 + r, n0 + c, e); partials(r, c); }
      }
      if (!in) continue;
      float v[4] = {f[0].x, f[0].y, f[0].z, f[0].w};
#pragma unroll
      for (int s = 1; s < 8; s++)
        if (s < split) { v[0] += f[s].x; v[1] += f[s].y; v[2] += f[s].z; v[3] += f[s].w; }
      epilogue4(p, m0 + r, n0 + c, v, e);
    }
    if (csum && tn == 0 && tid < rows) {
      const int r = first + tid;
      float w[8], v = 0.f;
#pragma unroll
      for (int s = 0; s < 8; s++)
        w[s] = s < split ? __uint_as_float(ld_cluster_u32(mapa_shared(csum_smem + (uint32_t)r * 4u, PAIR ? 2 * s + crank : s))) : 0.f;
#pragma unroll
      for (int s = 0; s < 8; s++)
        if (s < split) v += w[s];
      if (m0 + r < p.M) p.colsum[m0 + r] = p.accumulate ? p.colsum[m0 + r] + v : v;
    }
  }
  cluster_sync_all();                // no CTA leaves while another reads its partial tile
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem, BN); else tmem_dealloc(tmem, BN);
  }
}

// ------------------------------------------------------------------------------- launcher
static int g_num_sms = 0;
static int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

// Threads of a gemm_kernel CTA (or pair) that takes `turns` tiles.  Up to K = 1024 the main loop of a tile is shorter than the epilogue of four warps,
// which then bounds the product, and with one or two turns the last epilogue is a good part of it: eight warps.  us with eight / four, plain and with
// residual: K = 2048: 8192 x 512 14.5 / 14.9, 16.4 / 17.3; 8192 x 1024 24.8 / 25.0, 27.4 / 28.3; K = 4096: 4200 x 1024 25.4 / 27.3, 28.2 / 31.5; 4096 x 2048
// 46.2 / 46.5, 49.9 / 50.6; K = 6144: 1024 x 4096 35.5 / 35.8, 38.3 / 39.2.  Beyond, the epilogue hides behind the main loop and the second set of warps only
// takes power and issue slots from it (K = 8192: 8192 x 1024 100.2 / 97.7, 4200 x 1024 54.6 / 50.5, 1024 x 4096 48.2 / 48.5; 1.2B training step, K = 2048 and more
// in many turns: 147.3 ms with eight, 144.5 with four).
static int gemm_threads(const GemmParams& p, int turns) { return p.colsum || p.K <= 1024 || (turns <= 2 && p.K <= 6144) ? GEMM_THREADS : 192; }

// 256-row tiles on CTA pairs.  Returns the number of clusters that can be resident (0: unsupported).
static int g_pair_clusters = -1;
static int launch_gemm_pair(const CUtensorMap* ta, const CUtensorMap* tb, const GemmParams& p, int max_ctas, cudaStream_t st) {
  using Cfg = GemmCfg<256, true>;
  auto kern = gemm_kernel<256, true>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM; cfg.stream = st; cfg.attrs = attr;
  cfg.numAttrs = kh_pdl_enabled() ? 2 : 1;
  if (g_pair_clusters < 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
    if (e != cudaSuccess) { kh_set_error("gemm: cannot opt in to %d bytes of shared memory: %s", Cfg::SMEM, cudaGetErrorString(e)); return -1; }
    cfg.gridDim = dim3(2 * (num_sms() / 2));
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
    if (e != cudaSuccess || n < 1) { cudaGetLastError(); kh_set_error("gemm: CTA-pair launch is not available: %s", cudaGetErrorString(e)); g_pair_clusters = 0; return -1; }
    g_pair_clusters = n;
  }
  if (g_pair_clusters == 0) { kh_set_error("gemm: CTA-pair launch is not available"); return -1; }
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + 255) / 256);
  int clusters = tiles < g_pair_clusters ? tiles : g_pair_clusters;
  if (max_ctas > 0 && 2 * clusters > max_ctas) clusters = max_ctas / 2 > 0 ? max_ctas / 2 : 1;
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(gemm_threads(p, (tiles + clusters - 1) / clusters));
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, *ta, *tb, p);
  if (e != cudaSuccess) { kh_set_error("gemm pair launch failed: %s", cudaGetErrorString(e)); return -1; }
  return 0;
}
extern "C" int kh_gemm_pair_clusters() { return g_pair_clusters; }

template <int BN>
static int launch_gemm(const CUtensorMap* ta, const CUtensorMap* tb, const GemmParams& p, int max_ctas, cudaStream_t st) {
  using Cfg = GemmCfg<BN>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_kernel<BN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
    if (e != cudaSuccess) { kh_set_error("gemm: cannot opt in to %d bytes of shared memory: %s", Cfg::SMEM, cudaGetErrorString(e)); return -1; }
    attr_set = true;
  }
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  int grid = tiles < num_sms() ? tiles : num_sms();
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  cudaError_t e = KH_LAUNCH((gemm_kernel<BN, false>), grid, gemm_threads(p, (tiles + grid - 1) / grid), Cfg::SMEM, st, *ta, *tb, p);
  if (e != cudaSuccess) { kh_set_error("gemm launch failed: %s", cudaGetErrorString(e)); return -1; }
  return 0;
}

// Clusters of `split` CTAs (pairs: 2 split) that can be resident together (0: not available).
template <int BN, bool PAIR>
static int splitk_clusters(int split) {
  static int known[9] = {-1, -1, -1, -1, -1, -1, -1, -1, -1};
  int& n = known[split];
  if (n >= 0) return n;
  auto kern = gemm_splitk_kernel<BN, PAIR>;
  const int ctas = PAIR ? 2 * split : split;
  int got = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmCfg<BN, PAIR>::SMEM) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas * (num_sms() / ctas)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = GemmCfg<BN, PAIR>::SMEM;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&got, kern, &cfg) != cudaSuccess) got = 0;
  }
  cudaGetLastError();
  return n = got;
}
template <int BN, bool PAIR>
static int launch_splitk(const CUtensorMap* ta, const CUtensorMap* tb, const GemmParams& p, int split, cudaStream_t st) {
  if (splitk_clusters<BN, PAIR>(split) < 1) { kh_set_error("gemm: clusters of %d CTAs are not available", split); return -1; }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  const int ctas = PAIR ? 2 * split : split, tm = PAIR ? 2 * BM : BM;
  attr[0].val.clusterDim.x = ctas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(((p.M + tm - 1) / tm) * ((p.N + BN - 1) / BN) * ctas);
  cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = GemmCfg<BN, PAIR>::SMEM; cfg.stream = st;
  cfg.attrs = attr; cfg.numAttrs = kh_pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_splitk_kernel<BN, PAIR>, *ta, *tb, p, split);
  if (e != cudaSuccess) { kh_set_error("gemm split-K launch failed: %s", cudaGetErrorString(e)); return -1; }
  return 0;
}
// Tile width and split for a product that would take `chain` k-blocks one after the other on one CTA (0: no split).
// A split pays when the shortened chain saves more than the hand-off costs (SPLIT_COST k-blocks: 8 CTAs of 8 k-blocks take as
// long as one of 16 to 18); only splits whose tiles are all resident at once are taken (a second wave of clusters costs more
// than it saves: 1024 x 256 x 4096 in 4 x 64 12.2 us, in 8 x 64 25.7).
static int pick_splitk(int M, int N, int num_kb, int chain, int* bn_out) {
  constexpr int SPLIT_COST = 8, PAIR_COST = 14;
  const int tm = (M + BM - 1) / BM;
  int best = chain * 4 / 5, pick = 0;
  for (int bn = 128; bn >= 64; bn >>= 1)
    for (int split = 2; split <= 8; split <<= 1) {
      const int per = (num_kb + split - 1) / split, tiles = tm * ((N + bn - 1) / bn);
      if ((split - 1) * per >= num_kb || tiles * split > num_sms() || per + SPLIT_COST >= best) continue;
      if (tiles > (bn == 128 ? splitk_clusters<128, false>(split) : splitk_clusters<64, false>(split))) continue;
      best = per + SPLIT_COST; pick = split; *bn_out = bn;
    }
  // Pairs cover four times the output in a k-block; their launch and the sum of the larger tiles cost 6 k-blocks more (K = 9216: 1536 x 512 in 4 x 36
  // 21.8 us against 30.9 in 2 x 72, but 512 x 512 in 4 x 36 20.2 against 18.2 in 4 x 36 single CTAs).  Clusters of eight fit 15 times at most: 2048 x
  // 512, sixteen tiles, 27.3 in three slices, 39.1 in four.
  const int tiles2 = ((M + 255) / 256) * ((N + 255) / 256);
  if (M > 128 && N > 128)
    for (int split = 2; split <= 4; split++) {
      const int per = (num_kb + split - 1) / split;
      if ((split - 1) * per >= num_kb || tiles2 * 2 * split > num_sms() || per + PAIR_COST >= best) continue;
      if (tiles2 > splitk_clusters<256, true>(split)) continue;
      best = per + PAIR_COST; pick = split; *bn_out = 512;
    }
  return pick;
}

// C[M,N] = alpha * op(A) op(B) with a fused epilogue.  lda/ldb/ldc/ldaux are row pitches in
// elements of the row-major buffers described at the top of this file.  block_n = 0 lets the
// launcher pick the tile width (or a split of K over a cluster; 4096 * split + width asks for one, width 512 for pairs); max_ctas > 0 caps the grid (used to leave SMs to a
// concurrently running communication kernel).  Returns 0 or -1 (see kh_cuda_last_error).
//
// kh_gemm_bf16_colsum: same product with `colsum` [M] fp32 receiving colsum[m] (+)= sum_k op(A)[m, k]
// (`+=` when `accumulate`), computed from the A tiles in shared memory by four extra warps.  A must
// be in M-major form (a_mn), i.e. the call is a weight-gradient product dW = dY^T X and `colsum`
// is the bias gradient.
extern "C" int kh_gemm_bf16_colsum(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, void* C, int ldc,
                                   int M, int N, int K, int out_fp32, int accumulate, int epi, const void* bias, void* aux,
                                   int ldaux, float alpha, int block_n, int max_ctas, void* colsum, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) { kh_set_error("gemm: empty problem %dx%dx%d", M, N, K); return -1; }
  if (colsum && !a_mn) { kh_set_error("gemm: column sums need the A operand in M-major form"); return -1; }
  if (accumulate && !out_fp32) { kh_set_error("gemm: accumulate needs an fp32 output"); return -1; }
  if ((ldc % (out_fp32 ? 4 : 8)) != 0 || ((uintptr_t)C & 15)) { kh_set_error("gemm: output pitch/base not 16-byte aligned (ldc %d)", ldc); return -1; }
  if ((epi == EPI_BIAS || epi == EPI_BIAS_GELU || epi == EPI_BIAS_RESID || epi == EPI_GELU) && (!bias || ((uintptr_t)bias & 15))) { kh_set_error("gemm: bias missing or misaligned"); return -1; }
  if ((epi == EPI_BIAS_GELU || epi == EPI_BIAS_RESID || epi == EPI_DGELU || epi == EPI_RESID) && (!aux || (ldaux % 8) || ((uintptr_t)aux & 15))) { kh_set_error("gemm: aux operand missing or misaligned"); return -1; }
  int bn = block_n & 4095, split = block_n >> 12;
  const bool known_split = bn == 512 ? split >= 2 && split <= 4 : (split == 2 || split == 4 || split == 8) && (bn == 64 || bn == 128);
  if (split && (!known_split || (split - 1) * (((K + BK - 1) / BK + split - 1) / split) >= (K + BK - 1) / BK)) {
    kh_set_error("gemm: K split %d with tile width %d is not supported for K = %d", split, bn, K);
    return -1;
  }
  if (bn == 0) {
    // waves x relative tile time; narrower tiles reuse the A panel less and run at lower efficiency
    const int tm = (M + BM - 1) / BM, sms = num_sms();
    auto waves = [&](int w) { return (tm * ((N + w - 1) / w) + sms - 1) / sms; };
    // (up to K = 512 the epilogue weighs more and a 128-wide wave costs less: 8192 x 768 x 256 8.0 us in three waves of 128,
    // 8.8 in two of 256; 4096 x 1536 x 512 10.4 and 10.6; but with up to 64 rows half of the epilogue warps have nothing to do and
    // the main loop counts again: 16 x 50257 x 512 12.4 us in two waves of 256, 14.4 in three of 128; K = 256 8.6, 9.1 (64 rows 8.2, 8.1), K = 128 7.2, 7.0)
    const float c256 = waves(256) * 1.0f, c128 = waves(128) * (K <= (M > 64 ? 512 : 128) ? 0.62f : 0.7f), c64 = waves(64) * 0.5f;
    bn = 256;
    float best = c256;
    if (c128 < best) { best = c128; bn = 128; }
    if (c64 < best) { best = c64; bn = 64; }
    if (N <= 64) bn = 64;
    else if (N <= 128 && bn == 256) bn = 128;
    // 256 x 256 tiles on CTA pairs: a wave of pairs takes about 0.93 of a wave of single tiles
    // (measured 6-19 % faster on large shapes), so prefer it unless wave quantisation eats the gain.  A pair also pays about
    // 1 us for its cluster, which short main loops do not earn back: single tiles in up to four waves at K = 512
    // (9216 x 1536 14.3 us against 16.4; 8192 x 50257 in 86 waves 420 against 385), and up to K = 4096 where one wave does
    // (4200 x 1024, single tiles / pairs: K = 1024 11.2 / 12.2, 4096 26.8 / 27.5, 6144 42.8 / 40.1)
    if (bn == 256 && M >= 512 && g_pair_clusters != 0 && (waves(256) > (K <= 512 ? 4 : 1) || K > 4096)) {
      const int clusters = g_pair_clusters > 0 ? g_pair_clusters : sms / 2;
      const int tiles2 = ((M + 255) / 256) * ((N + 255) / 256);
      const float cpair = (float)((tiles2 + clusters - 1) / clusters) * 0.93f;
      if (cpair <= best) bn = 512;
    }
    if (max_ctas == 0) {
      const int num_kb = (K + BK - 1) / BK, workers = bn == 512 ? sms / 2 : sms;
      const int tiles = bn == 512 ? ((M + 255) / 256) * ((N + 255) / 256) : tm * ((N + bn - 1) / bn);
      split = pick_splitk(M, N, num_kb, (tiles + workers - 1) / workers * num_kb, &bn);
    }
  }
  const bool pair = bn == 512;                  // 256 x 256 tiles on CTA pairs (cta_group::2)
  if (pair) bn = 256;
  if (bn != 64 && bn != 128 && bn != 256) { kh_set_error("gemm: block_n must be 64, 128, 256 or 512 (CTA pairs)"); return -1; }
  const CUtensorMap* ta = a_mn ? kh_tmap_2d_bf16(A, K, M, lda, BK, 64) : kh_tmap_2d_bf16(A, M, K, lda, BM, BK);
  if (!ta) return -1;
  const CUtensorMap* tb = b_mn ? kh_tmap_2d_bf16(B, K, N, ldb, BK, 64) : kh_tmap_2d_bf16(B, N, K, ldb, pair ? 128 : bn, BK);
  if (!tb) return -1;
  GemmParams p;
  p.M = M; p.N = N; p.K = K; p.a_mn = a_mn; p.b_mn = b_mn; p.C = C; p.ldc = ldc; p.out_fp32 = out_fp32;
  p.accumulate = accumulate; p.epi = epi; p.bias = (const bf16*)bias; p.aux = (bf16*)aux; p.ldaux = ldaux; p.alpha = alpha;
  p.colsum = (float*)colsum;
  p.err = kh_error_word_dev();
  cudaStream_t st = (cudaStream_t)stream;
  if (split && pair) return launch_splitk<256, true>(ta, tb, p, split, st);
  if (split) return bn == 128 ? launch_splitk<128, false>(ta, tb, p, split, st) : launch_splitk<64, false>(ta, tb, p, split, st);
  if (pair) return launch_gemm_pair(ta, tb, p, max_ctas, st);
  if (bn == 256) return launch_gemm<256>(ta, tb, p, max_ctas, st);
  if (bn == 128) return launch_gemm<128>(ta, tb, p, max_ctas, st);
  return launch_gemm<64>(ta, tb, p, max_ctas, st);
}

extern "C" int kh_gemm_bf16(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, void* C, int ldc,
                            int M, int N, int K, int out_fp32, int accumulate, int epi, const void* bias, void* aux,
                            int ldaux, float alpha, int block_n, int max_ctas, void* stream) {
  return kh_gemm_bf16_colsum(A, lda, a_mn, B, ldb, b_mn, C, ldc, M, N, K, out_fp32, accumulate, epi, bias, aux, ldaux,
                             alpha, block_n, max_ctas, nullptr, stream);
}
