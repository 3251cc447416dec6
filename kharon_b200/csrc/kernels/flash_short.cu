// Causal attention of short sequences (T <= 64), forward and backward: one CTA per (batch, head).
//
// The tcgen05 kernels work on tiles of 128 rows.  A policy update on 512 samples of 18 tokens is 4096 (batch, head) items of one
// tile, 14 % of it rows: each item pays the whole TMA -> tcgen05.mma -> TMEM -> store chain for 18 rows, and what bounds it is
// that latency times 14 items per resident CTA, not the 75 MB it moves.  Here Q, K, V (and dO) of an item sit in shared memory
// (rows padded by 16 bytes: conflict-free ldmatrix), a warp owns 16 rows and multiplies them with mma.sync m16n8k16, scores
// and probabilities never leave its registers, and several CTAs per SM hide each other's loads.
//   forward   warp = 16 queries: S = Q K^T, softmax, O = P V
//   backward  warps 0 .. RT-1 = 16 queries each: dQ = dS K;  warps RT .. 2RT-1 = 16 keys each, with everything transposed:
//             S^T = K Q^T, dP^T = V dO^T, dV = P^T dO, dK = dS^T Q.  S is formed twice, every gradient has one writer.
// Rounding points are those of the tcgen05 kernels: fp32 scores and statistics, P and dS rounded to bf16 for their products,
// the normaliser applied to the fp32 result.
#include "common.cuh"

#include "flash_short.h"

namespace {

constexpr float LOG2E = 1.4426950408889634f;
static_assert(KH_FLASH_SHORT_T == 64, "one to four row tiles of 16");

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// [rows x HD] matrix in shared memory, pitch HD + 8
template <int HD> struct Tile {
  static constexpr int PITCH = (HD + 8) * 2;
  // 16 x 16 block as A operand (rows r0.., columns c0..)
  static __device__ __forceinline__ uint32_t a(uint32_t base, int lane, int r0, int c0) {
    return base + (r0 + (lane & 15)) * PITCH + (c0 + (lane >> 4) * 8) * 2;
  }
  // 16 rows x 16 columns as two B operands (columns of the product = rows r0.. and r0 + 8.., contraction over columns c0..)
  static __device__ __forceinline__ uint32_t b(uint32_t base, int lane, int r0, int c0) {
    return base + (r0 + (lane & 7) + (lane >> 4) * 8) * PITCH + (c0 + ((lane >> 3) & 1) * 8) * 2;
  }
  // same block, contraction over rows r0.., columns of the product = columns c0.. and c0 + 8.. (transposing load)
  static __device__ __forceinline__ uint32_t bt(uint32_t base, int lane, int r0, int c0) {
    return base + (r0 + (lane & 15)) * PITCH + (c0 + (lane >> 4) * 8) * 2;
  }
};
// rows [0, T) of a matrix with row pitch `ld` -> shared memory, rows [T, rows) zero.  Asynchronous: what bounds these kernels is the way
// from memory into the tiles and out of them, so all loads of a CTA are in flight at once and
// rows leave in pieces of 16 bytes (B 512 H 8 T 18 head width 64: backward 36.2 us with one load after the other and words of 4 bytes, 25.2 so, forward
// 11.4 and 10.8; B 256 H 16 T 64: 174 and 99.9, 35.6 and 25.3; head width 128, B 512 H 8 T 18: 77.1 and 55.4, 23.3 and 17.8).
template <int HD>
__device__ __forceinline__ void load_rows(uint32_t dst, const bf16* src, size_t ld, int T, int rows) {
  for (int i = threadIdx.x; i < rows * (HD / 8); i += blockDim.x) {
    const int r = i / (HD / 8), c = i % (HD / 8);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * Tile<HD>::PITCH + c * 16),
                 "l"(src + (r < T ? (size_t)r * ld : 0) + c * 8), "r"(r < T ? 16 : 0) : "memory");
  }
}
__device__ __forceinline__ void load_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// acc[16 x 8 nt] = rows r0.. of X times rows 0.. of Y transposed (nt column tiles of 8, only tiles [lo, hi) are formed)
template <int HD, int RT>
__device__ __forceinline__ void scores(float (&acc)[2 * RT][4], uint32_t X, uint32_t Y, int lane, int r0, int lo, int hi) {
#pragma unroll
  for (int t = 0; t < 2 * RT; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[t][i] = 0.f;
#pragma unroll
  for (int k = 0; k < HD; k += 16) {
    uint32_t a[4];
    ldsm4(a, Tile<HD>::a(X, lane, r0, k));
#pragma unroll
    for (int t = 0; t < RT; t++)
      if (2 * t >= lo && 2 * t < hi) {
        uint32_t b[4];
        ldsm4(b, Tile<HD>::b(Y, lane, t * 16, k));
        mma(acc[2 * t], a, b[0], b[1]);
        mma(acc[2 * t + 1], a, b[2], b[3]);
      }
  }
}
// acc[16 x HD] += P[16 x 16 t] times rows of Y (tiles [lo, hi) of P, in bf16)
template <int HD, int RT>
__device__ __forceinline__ void accumulate(float (&acc)[HD / 8][4], const float (&p)[2 * RT][4], uint32_t Y, int lane, int lo, int hi) {
#pragma unroll
  for (int t = 0; t < RT; t++)
    if (2 * t >= lo && 2 * t < hi) {
      const uint32_t a[4] = {pack_bf16(p[2 * t][0], p[2 * t][1]), pack_bf16(p[2 * t][2], p[2 * t][3]),
                             pack_bf16(p[2 * t + 1][0], p[2 * t + 1][1]), pack_bf16(p[2 * t + 1][2], p[2 * t + 1][3])};
#pragma unroll
      for (int c = 0; c < HD; c += 16) {
        uint32_t b[4];
        ldsm4t(b, Tile<HD>::bt(Y, lane, t * 16, c));
        mma(acc[c / 8], a, b[0], b[1]);
        mma(acc[c / 8 + 1], a, b[2], b[3]);
      }
    }
}
// The four lanes of a row hold two columns of every tile of eight; lane q gets all columns of tile q (of four tiles).
__device__ __forceinline__ uint4 own_tile(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, int lane) {
  const bool odd = lane & 1, high = lane & 2;
  const uint32_t x = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 1), y = __shfl_xor_sync(0xffffffffu, odd ? a2 : a3, 1);
  const uint32_t p0 = odd ? x : a0, p1 = odd ? a1 : x, s0 = odd ? y : a2, s1 = odd ? a3 : y;      // tiles (q & 1) and (q & 1) + 2 of two lanes
  const uint32_t u = __shfl_xor_sync(0xffffffffu, high ? p0 : s0, 2), v = __shfl_xor_sync(0xffffffffu, high ? p1 : s1, 2);
  return high ? make_uint4(u, v, s0, s1) : make_uint4(p0, p1, u, v);
}
template <int HD>
__device__ __forceinline__ void store(bf16* dst, size_t ld, const float (&acc)[HD / 8][4], float m0, float m1, int lane, int r0, int T) {
  const int g = lane >> 2, c = (lane & 3) * 8;
#pragma unroll
  for (int t = 0; t < HD / 8; t += 4) {
    uint32_t w[4], z[4];
#pragma unroll
    for (int i = 0; i < 4; i++) { w[i] = pack_bf16(acc[t + i][0] * m0, acc[t + i][1] * m0); z[i] = pack_bf16(acc[t + i][2] * m1, acc[t + i][3] * m1); }
    const uint4 lo = own_tile(w[0], w[1], w[2], w[3], lane), hi = own_tile(z[0], z[1], z[2], z[3], lane);
    if (r0 + g < T) *reinterpret_cast<uint4*>(dst + (size_t)(r0 + g) * ld + t * 8 + c) = lo;
    if (r0 + g + 8 < T) *reinterpret_cast<uint4*>(dst + (size_t)(r0 + g + 8) * ld + t * 8 + c) = hi;
  }
}

template <int HD, int RT>
__global__ void __launch_bounds__(32 * RT)
flash_short_fwd_k(const bf16* __restrict__ qkv, int ld, bf16* __restrict__ out, float* __restrict__ lse, int T, int H, float scale) {
  extern __shared__ __align__(16) uint8_t smem[];
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.x / H, h = blockIdx.x % H, d = H * HD;
  constexpr int rows = 16 * RT;
  const uint32_t sQ = smem_u32(smem), sK = sQ + rows * Tile<HD>::PITCH, sV = sK + rows * Tile<HD>::PITCH;
  const bf16* src = qkv + (size_t)b * T * ld + h * HD;
  load_rows<HD>(sQ, src, ld, T, rows);
  load_rows<HD>(sK, src + d, ld, T, rows);
  load_rows<HD>(sV, src + 2 * d, ld, T, rows);
  load_wait();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r0 = warp * 16, g = lane >> 2, c = (lane & 3) * 2;
  const int hi = 2 * (warp + 1);                   // column tiles up to the diagonal
  float s[2 * RT][4];
  scores<HD, RT>(s, sQ, sK, lane, r0, 0, hi);
  const float sl2 = scale * LOG2E;
  float mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int t = 0; t < 2 * RT; t++)
    if (t < hi)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (t * 8 + c + (i & 1) > r0 + g + (i >> 1) * 8) s[t][i] = -INFINITY;
        mx[i >> 1] = fmaxf(mx[i >> 1], s[t][i]);
      }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2)) * sl2;
  }
#pragma unroll
  for (int t = 0; t < 2 * RT; t++)
    if (t < hi)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        s[t][i] = exp2f(fmaf(s[t][i], sl2, -mx[i >> 1]));
        l[i >> 1] += s[t][i];
      }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
  float o[HD / 8][4];
#pragma unroll
  for (int t = 0; t < HD / 8; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[t][i] = 0.f;
  accumulate<HD, RT>(o, s, sV, lane, 0, hi);
  store<HD>(out + (size_t)b * T * d + h * HD, d, o, 1.f / l[0], 1.f / l[1], lane, r0, T);
  if (lse && (lane & 3) == 0) {
    float* q = lse + ((size_t)b * H + h) * T;
    if (r0 + g < T) q[r0 + g] = (mx[0] + log2f(l[0])) / LOG2E;
    if (r0 + g + 8 < T) q[r0 + g + 8] = (mx[1] + log2f(l[1])) / LOG2E;
  }
}

template <int HD, int RT>
__global__ void __launch_bounds__(64 * RT)
flash_short_bwd_k(const bf16* __restrict__ qkv, int ld, const bf16* __restrict__ out, const bf16* __restrict__ dout,
                  const float* __restrict__ lse, bf16* __restrict__ dqkv, float* __restrict__ delta, int T, int H, float scale) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float s_lse[16 * RT], s_delta[16 * RT];
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.x / H, h = blockIdx.x % H, d = H * HD;
  constexpr int rows = 16 * RT;
  const uint32_t sQ = smem_u32(smem), sK = sQ + rows * Tile<HD>::PITCH, sV = sK + rows * Tile<HD>::PITCH, sD = sV + rows * Tile<HD>::PITCH;
  const bf16* src = qkv + (size_t)b * T * ld + h * HD;
  const bf16* dsrc = dout + (size_t)b * T * d + h * HD;
  const bf16* osrc = out + (size_t)b * T * d + h * HD;
  load_rows<HD>(sQ, src, ld, T, rows);
  load_rows<HD>(sK, src + d, ld, T, rows);
  load_rows<HD>(sV, src + 2 * d, ld, T, rows);
  load_rows<HD>(sD, dsrc, d, T, rows);
  // delta = rowsum(dO * O): HD / 8 lanes per row, as in the kernel for long sequences
  // each thread takes the pieces of dO that it loaded itself
  constexpr int LPH = HD / 8, OWN = 16 * LPH / 64;
  uint4 x[OWN];
  float l[OWN];
#pragma unroll
  for (int k = 0; k < OWN; k++) {
    const int i = threadIdx.x + k * 64 * RT, r = i / LPH, c = i % LPH;
    x[k] = make_uint4(0, 0, 0, 0);
    l[k] = INFINITY;
    if (r < T) {
      x[k] = *reinterpret_cast<const uint4*>(osrc + (size_t)r * d + c * 8);
      if (c == 0) l[k] = lse[((size_t)b * H + h) * T + r];
    }
  }
  load_wait();
#pragma unroll
  for (int k = 0; k < OWN; k++) {
    const int i = threadIdx.x + k * 64 * RT, r = i / LPH, c = i % LPH;
    uint4 y;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w) : "r"(sD + r * Tile<HD>::PITCH + c * 16) : "memory");
    const float2 x0 = unpack_bf16(x[k].x), x1 = unpack_bf16(x[k].y), x2 = unpack_bf16(x[k].z), x3 = unpack_bf16(x[k].w);
    const float2 y0 = unpack_bf16(y.x), y1 = unpack_bf16(y.y), y2 = unpack_bf16(y.z), y3 = unpack_bf16(y.w);
    float s = (x0.x * y0.x + x0.y * y0.y) + (x1.x * y1.x + x1.y * y1.y) + (x2.x * y2.x + x2.y * y2.y) + (x3.x * y3.x + x3.y * y3.y);
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (c == 0) {
      s_delta[r] = s;
      s_lse[r] = l[k] * LOG2E;
      if (r < T) delta[((size_t)b * H + h) * T + r] = s;
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = (lane & 3) * 2;
  const float sl2 = scale * LOG2E;
  bf16* dst = dqkv + (size_t)b * T * ld + h * HD;
  float s[2 * RT][4], dp[2 * RT][4];
  float acc[HD / 8][4];
#pragma unroll
  for (int t = 0; t < HD / 8; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[t][i] = 0.f;
  if (warp < RT) {                                 // 16 queries, keys up to the diagonal
    const int r0 = warp * 16, hi = 2 * (warp + 1);
    scores<HD, RT>(s, sQ, sK, lane, r0, 0, hi);
    scores<HD, RT>(dp, sD, sV, lane, r0, 0, hi);
    const float ls[2] = {s_lse[r0 + g], s_lse[r0 + g + 8]}, de[2] = {s_delta[r0 + g], s_delta[r0 + g + 8]};
#pragma unroll
    for (int t = 0; t < 2 * RT; t++)
      if (t < hi)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          float p = exp2f(fmaf(s[t][i], sl2, -ls[i >> 1]));
          if (t * 8 + c + (i & 1) > r0 + g + (i >> 1) * 8) p = 0.f;
          s[t][i] = p * (dp[t][i] - de[i >> 1]) * scale;
        }
    accumulate<HD, RT>(acc, s, sK, lane, 0, hi);
    store<HD>(dst, ld, acc, 1.f, 1.f, lane, r0, T);
  } else {                                         // 16 keys, queries from the diagonal on
    const int r0 = (warp - RT) * 16, lo = 2 * (warp - RT), hi = 2 * RT;
    scores<HD, RT>(s, sK, sQ, lane, r0, lo, hi);
#pragma unroll
    for (int t = 0; t < 2 * RT; t++)
      if (t >= lo && t < hi)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int q = t * 8 + c + (i & 1);
          float p = exp2f(fmaf(s[t][i], sl2, -s_lse[q]));
          if (r0 + g + (i >> 1) * 8 > q) p = 0.f;
          s[t][i] = p;
        }
    accumulate<HD, RT>(acc, s, sD, lane, lo, hi);
    store<HD>(dst + 2 * d, ld, acc, 1.f, 1.f, lane, r0, T);
    scores<HD, RT>(dp, sV, sD, lane, r0, lo, hi);
#pragma unroll
    for (int t = 0; t < 2 * RT; t++)
      if (t >= lo && t < hi)
#pragma unroll
        for (int i = 0; i < 4; i++) s[t][i] = s[t][i] * (dp[t][i] - s_delta[t * 8 + c + (i & 1)]) * scale;
#pragma unroll
    for (int t = 0; t < HD / 8; t++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[t][i] = 0.f;
    accumulate<HD, RT>(acc, s, sQ, lane, lo, hi);
    store<HD>(dst + d, ld, acc, 1.f, 1.f, lane, r0, T);
  }
}

int check(const void* p, long ld, const char* what) {
  if (((uintptr_t)p & 15) || (ld % 8)) { kh_set_error("flash: %s needs a 16-byte aligned base and row pitch (ld %ld)", what, ld); return -1; }
  return 0;
}
template <typename K>
int opt_in(K kernel, int bytes) {
  if (bytes <= 48 * 1024) return 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess) return 0;
  kh_set_error("flash: cannot opt in to %d bytes of shared memory", bytes);
  return -1;
}
template <int HD, int RT>
int fwd(const bf16* qkv, bf16* out, float* lse, int B, int T, int H, int ld, float scale, cudaStream_t st) {
  const int smem = 3 * RT * 16 * Tile<HD>::PITCH;
  if (opt_in(flash_short_fwd_k<HD, RT>, smem)) return -1;
  if (KH_LAUNCH((flash_short_fwd_k<HD, RT>), B * H, 32 * RT, smem, st, qkv, ld, out, lse, T, H, scale) != cudaSuccess) { kh_set_error("flash_short_fwd: launch failed"); return -1; }
  return 0;
}
template <int HD, int RT>
int bwd(const bf16* qkv, const bf16* out, const bf16* dout, const float* lse, bf16* dqkv, float* delta, int B, int T, int H, int ld,
        float scale, cudaStream_t st) {
  const int smem = 4 * RT * 16 * Tile<HD>::PITCH;
  if (opt_in(flash_short_bwd_k<HD, RT>, smem)) return -1;
  if (KH_LAUNCH((flash_short_bwd_k<HD, RT>), B * H, 64 * RT, smem, st, qkv, ld, out, dout, lse, dqkv, delta, T, H, scale) != cudaSuccess) { kh_set_error("flash_short_bwd: launch failed"); return -1; }
  return 0;
}
#define BY_ROWS(FN, HD, ...) (T <= 16 ? FN<HD, 1>(__VA_ARGS__) : T <= 32 ? FN<HD, 2>(__VA_ARGS__) : T <= 48 ? FN<HD, 3>(__VA_ARGS__) : FN<HD, 4>(__VA_ARGS__))

}  // namespace

int kh_flash_short_fwd(const void* qkv, void* out, void* lse, int B, int T, int H, int hd, int ld, float scale, void* stream) {
  if (check(qkv, ld, "qkv") || check(out, 0, "out")) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  return hd == 64 ? BY_ROWS(fwd, 64, (const bf16*)qkv, (bf16*)out, (float*)lse, B, T, H, ld, scale, st)
                  : BY_ROWS(fwd, 128, (const bf16*)qkv, (bf16*)out, (float*)lse, B, T, H, ld, scale, st);
}
int kh_flash_short_bwd(const void* qkv, const void* out, const void* dout, const void* lse, void* dqkv, void* delta, int B, int T,
                       int H, int hd, int ld, float scale, void* stream) {
  if (check(qkv, ld, "qkv") || check(out, 0, "out") || check(dout, 0, "dout") || check(dqkv, ld, "dqkv")) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  return hd == 64 ? BY_ROWS(bwd, 64, (const bf16*)qkv, (const bf16*)out, (const bf16*)dout, (const float*)lse, (bf16*)dqkv, (float*)delta, B, T, H, ld, scale, st)
                  : BY_ROWS(bwd, 128, (const bf16*)qkv, (const bf16*)out, (const bf16*)dout, (const float*)lse, (bf16*)dqkv, (float*)delta, B, T, H, ld, scale, st);
}
