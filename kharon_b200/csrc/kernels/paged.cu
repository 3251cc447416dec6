// Paged-KV inference kernels: KV append, paged attention over block tables, last-row gather,
// KV block copy (copy-on-write) and the on-device sampler.
//
// KV pool of one layer: k, v : [n_blocks, block_size, H, hd] bf16 (reference src/core/infer.c:20-21
// keeps [n_layer, n_blocks, bs, H, hd]; here the layer is the outermost index of the same
// allocation, the caller passes the layer's base pointer).  A step carries a flat token list
// (pos[i], slot[i]) and a dense block table [n_seq, max_lb] exactly as infer.c:229-249.
//
// Replaces src/kernels/paged.cu: append_kv_k :33-46, paged_attn_k :50-77 (one key per block-wide
// tree reduction), gather_rows_k :80-86, and the host sampler infer.c:197-213.
#include "common.cuh"

#define KH_LAUNCH_CHECK(name)                                                     \
  do {                                                                            \
    cudaError_t e_ = cudaGetLastError();                                          \
    if (e_ != cudaSuccess) { kh_set_error(name ": %s", cudaGetErrorString(e_)); return -1; } \
  } while (0)

static inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// ------------------------------------------------------------------------------- append
// One thread per 8 elements: copies k and v of every new token into its block slot.
__global__ void append_kv_k(const bf16* __restrict__ qkv, int ld, bf16* __restrict__ kc, bf16* __restrict__ vc,
                            const int* __restrict__ pos, const int* __restrict__ slot, const int* __restrict__ btab,
                            int max_lb, int bs, int d, int ntok, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  const int per = d / 8;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)ntok * per) return;
  const int t = (int)(i / per), c = (int)(i % per) * 8;
  const int p = pos[t];
  // index guard: a position beyond the block table is recorded (status code 8) and its store skipped
  if (p < 0 || p / bs >= max_lb || slot[t] < 0) { atomicCAS(err, 0, 8); return; }
  const int blk = btab[(size_t)slot[t] * max_lb + p / bs];
  const size_t dst = ((size_t)blk * bs + (p % bs)) * d + c;
  const bf16* src = qkv + (size_t)t * ld;
  *reinterpret_cast<uint4*>(kc + dst) = *reinterpret_cast<const uint4*>(src + d + c);
  *reinterpret_cast<uint4*>(vc + dst) = *reinterpret_cast<const uint4*>(src + 2 * d + c);
}
extern "C" int kh_append_kv(const void* qkv, int ld, void* kc, void* vc, const void* pos, const void* slot,
                            const void* btab, int max_lb, int bs, int H, int hd, int ntok, void* stream) {
  const int d = H * hd;
  if (d % 8) { kh_set_error("append_kv: H*hd must be a multiple of 8"); return -1; }
  KH_LAUNCH(append_kv_k, cdiv((long)ntok * d / 8, 256), 256, 0, (cudaStream_t)stream, 
      (const bf16*)qkv, ld, (bf16*)kc, (bf16*)vc, (const int*)pos, (const int*)slot, (const int*)btab, max_lb, bs, d, ntok,
      kh_error_word_dev());
  KH_LAUNCH_CHECK("append_kv");
  return 0;
}

// ------------------------------------------------------------------------------- attention
// W warps per (token, head) item, 4 / W items per CTA of four warps.  A key or value row is read by HD / 8 lanes in 16-byte
// pieces, so a warp holds 256 / HD lane groups; group i of an item takes keys i, i + ST, i + 2 ST, ... (ST = W * 256 / HD),
// four at a time, with a running fp32 softmax of its own, and the groups are merged once at the end (shuffles in the warp,
// shared memory in warp order across warps).  K and V of a position are fetched together, and the next four positions replace
// the current ones in their registers as soon as those are used: one trip to memory per four keys and no CTA barrier in the
// loop.  Neighbouring items are tokens of the same head, which read mostly the same rows (L1).
// W = 1 when the items fill the chip by themselves (prefill, large batches), else 4, and 2 between for narrow heads (8 heads of 32,
// 128 tokens, us with W = 1 / 2 / 4: context 20 3.7 / 4.1 / 6.3, context 200 10.1 / 8.8 / 10.7, context 1000 41.7 / 31.1 / 32.6).
// A CTA of 128 threads per item with barriers between scores, maximum, sum and value passes took 25.6 us for 512 tokens x 8
// heads at contexts of 9 to 18.
// Context = positions 0..pos of the token's own sequence.  With `append` != 0 (decode steps: one new token per sequence) the
// group that owns position pos takes the token's k and v from the qkv row and writes them into the cache; otherwise
// the new tokens' K/V must already be in the cache (prefill: several tokens of one sequence attend to each other).
template <int HD, int W>
__global__ void __launch_bounds__(128)
paged_attn_k(const bf16* __restrict__ qkv, int ld, bf16* kc, bf16* vc, bf16* __restrict__ out, const int* __restrict__ pos,
             const int* __restrict__ slot, const int* __restrict__ btab, int max_lb, int bs, int H, int ntok, float scale,
             int max_ctx, int append, int vec, int* err) {
  constexpr int LPK = HD / 8, KPW = 32 / LPK, ST = W * KPW, IPC = 4 / W;      // lanes per key, keys per warp, items per CTA
  __shared__ float s_part[W > 1 ? 4 * (HD + 2) : 1];
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = (int)blockIdx.x * IPC + warp / W, h = blockIdx.y, wi = warp % W;
  const int kg = wi * KPW + lane / LPK, e0 = (lane % LPK) * 8, d = H * HD;
  const bool live = t < ntok;
  const int p = live ? pos[t] : -1, sl = live ? slot[t] : -1;
  // index guard: a context longer than the caller's limit or the block table is recorded (status code 8) and the token skipped
  const bool valid = live && p >= 0 && p < max_ctx && p / bs < max_lb && sl >= 0;        // uniform over the item's warps
  if (live && !valid && lane == 0) atomicCAS(err, 0, 8);
  float m = -INFINITY, l = 0.f, o[8];
#pragma unroll
  for (int k = 0; k < 8; k++) o[k] = 0.f;
  if (valid) {
    const bf16* row = qkv + (size_t)t * ld + h * HD + e0;
    const int* bt = btab + (size_t)sl * max_lb;
    const int n = append ? p : p + 1;              // positions read from the cache
    auto at = [&](int j) { return ((size_t)__ldg(bt + j / bs) * bs + (j % bs)) * d + h * HD + e0; };
    uint4 k4[4], v4[4], kn = make_uint4(0, 0, 0, 0), vn = kn;
    size_t a4[4];
    auto rows = [&](int j0) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (j0 + i * ST < n) a4[i] = at(j0 + i * ST);
    };
    auto fetch = [&](uint4 (&r)[4], const bf16* c, int j0) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (j0 + i * ST < n) r[i] = *reinterpret_cast<const uint4*>(c + a4[i]);
    };
    rows(kg);
    fetch(k4, kc, kg);
    fetch(v4, vc, kg);
    rows(kg + 4 * ST);
    if (append && p % ST == kg) {
      kn = *reinterpret_cast<const uint4*>(row + d);
      vn = *reinterpret_cast<const uint4*>(row + 2 * d);
      *reinterpret_cast<uint4*>(kc + at(p)) = kn;
      *reinterpret_cast<uint4*>(vc + at(p)) = vn;
    }
    float q[8];
    {
      uint4 u;
      if (vec) u = *reinterpret_cast<const uint4*>(row);
      else {                                       // rows that are not 16-byte aligned
        uint16_t e16[8];
        for (int k = 0; k < 8; k++) e16[k] = reinterpret_cast<const uint16_t*>(row)[k];
        u = make_uint4(e16[0] | (uint32_t)e16[1] << 16, e16[2] | (uint32_t)e16[3] << 16, e16[4] | (uint32_t)e16[5] << 16, e16[6] | (uint32_t)e16[7] << 16);
      }
      const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), e = unpack_bf16(u.w);
      q[0] = a.x * scale; q[1] = a.y * scale; q[2] = b.x * scale; q[3] = b.y * scale;
      q[4] = c.x * scale; q[5] = c.y * scale; q[6] = e.x * scale; q[7] = e.y * scale;
    }
#pragma unroll 1
    for (int b0 = 0; wi * KPW + b0 <= p; b0 += 4 * ST) {          // uniform over the warp
      const int j0 = kg + b0;
      float s[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int j = j0 + i * ST;
        if (j >= n) { k4[i] = kn; v4[i] = vn; }                   // the appended position, or past the end (masked below)
        const float2 a = unpack_bf16(k4[i].x), b = unpack_bf16(k4[i].y), c = unpack_bf16(k4[i].z), e = unpack_bf16(k4[i].w);
        s[i] = a.x * q[0] + a.y * q[1] + b.x * q[2] + b.y * q[3] + c.x * q[4] + c.y * q[5] + e.x * q[6] + e.y * q[7];
      }
      fetch(k4, kc, j0 + 4 * ST);
#pragma unroll
      for (int x = LPK / 2; x > 0; x >>= 1)
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] += __shfl_xor_sync(0xffffffffu, s[i], x);
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (j0 + i * ST > p) { s[i] = -INFINITY; v4[i] = make_uint4(0, 0, 0, 0); }
      const float mn = fmaxf(m, fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3])));
      const float ref = mn == -INFINITY ? 0.f : mn;
      const float sc = __expf(m - ref);
      m = mn;
      l *= sc;
#pragma unroll
      for (int k = 0; k < 8; k++) o[k] *= sc;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float pr = __expf(s[i] - ref);
        l += pr;
        const float2 a = unpack_bf16(v4[i].x), b = unpack_bf16(v4[i].y), c = unpack_bf16(v4[i].z), e = unpack_bf16(v4[i].w);
        o[0] += pr * a.x; o[1] += pr * a.y; o[2] += pr * b.x; o[3] += pr * b.y;
        o[4] += pr * c.x; o[5] += pr * c.y; o[6] += pr * e.x; o[7] += pr * e.y;
      }
      fetch(v4, vc, j0 + 4 * ST);
      rows(j0 + 8 * ST);
    }
#pragma unroll
    for (int x = LPK; x < 32; x <<= 1) {            // merge the lane groups of the warp
      const float m2 = __shfl_xor_sync(0xffffffffu, m, x), l2 = __shfl_xor_sync(0xffffffffu, l, x);
      const float mn = fmaxf(m, m2), ref = mn == -INFINITY ? 0.f : mn;
      const float c1 = __expf(m - ref), c2 = __expf(m2 - ref);
      m = mn;
      l = l * c1 + l2 * c2;
#pragma unroll
      for (int k = 0; k < 8; k++) o[k] = o[k] * c1 + __shfl_xor_sync(0xffffffffu, o[k], x) * c2;
    }
  }
  if (W > 1) {                                      // merge an item's warps in order; the first one writes
    float* part = s_part + warp * (HD + 2);
    if (lane < LPK) {
#pragma unroll
      for (int k = 0; k < 8; k++) part[e0 + k] = o[k];
      if (lane == 0) { part[HD] = m; part[HD + 1] = l; }
    }
    __syncthreads();
    if (wi != 0 || !valid) return;
    const float* parts = s_part + warp * (HD + 2);
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < W; w++) mx = fmaxf(mx, parts[w * (HD + 2) + HD]);
    l = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) o[k] = 0.f;
#pragma unroll
    for (int w = 0; w < W; w++) {
      const float c = __expf(parts[w * (HD + 2) + HD] - mx);      // (position 0 is always there: mx is finite or NaN)
      l += c * parts[w * (HD + 2) + HD + 1];
#pragma unroll
      for (int k = 0; k < 8; k++) o[k] += c * parts[w * (HD + 2) + e0 + k];
    }
  }
  if (valid && lane < LPK) {
    const float inv = 1.f / l;
    bf16* dst = out + (size_t)t * d + h * HD + e0;
    if (!vec)
      for (int k = 0; k < 8; k++) dst[k] = __float2bfloat16(o[k] * inv);
    else *reinterpret_cast<uint4*>(dst) =
        make_uint4(pack_bf16(o[0] * inv, o[1] * inv), pack_bf16(o[2] * inv, o[3] * inv), pack_bf16(o[4] * inv, o[5] * inv),
                   pack_bf16(o[6] * inv, o[7] * inv));
  }
}
extern "C" int kh_paged_attn(const void* qkv, int ld, void* kc, void* vc, void* out, const void* pos,
                             const void* slot, const void* btab, int max_lb, int bs, int H, int hd, float scale,
                             int ntok, int max_ctx, int append, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  // one range per token ends at some 50000 positions; longer contexts belong to kh_paged_attn_split
  if ((size_t)(hd + max_ctx + 1024 + 8) * sizeof(float) > 200 * 1024) { kh_set_error("paged_attn: context %d is too long for one range", max_ctx); return -1; }
  const int vec = ((uintptr_t)qkv & 15) == 0 && ((uintptr_t)out & 15) == 0 && ld % 8 == 0;
  // one warp per item once the items alone give every SM some sixteen warps, else four; two for narrow heads, whose warp covers 32
  // (64) positions a turn, once four would not fit the chip together
  const long items = (long)ntok * H;
  const int W = items >= 148 * 16 ? 1 : hd <= 32 && items > 148 * 4 ? 2 : 4;
#define LAUNCH_W(HD, W)                                                                                                     \
  KH_LAUNCH((paged_attn_k<HD, W>), dim3(cdiv((long)ntok * W, 4), H), 128, 0, st, (const bf16*)qkv, ld, (bf16*)kc, (bf16*)vc, \
            (bf16*)out, (const int*)pos, (const int*)slot, (const int*)btab, max_lb, bs, H, ntok, scale, max_ctx, append, vec, \
            kh_error_word_dev())
#define LAUNCH(HD) { if (W == 1) LAUNCH_W(HD, 1); else LAUNCH_W(HD, 4); }
#define LAUNCH_NARROW(HD) { if (W == 2) LAUNCH_W(HD, 2); else LAUNCH(HD) }
  if (hd == 128) LAUNCH(128)
  else if (hd == 64) LAUNCH(64)
  else if (hd == 32) LAUNCH_NARROW(32)
  else if (hd == 16) LAUNCH_NARROW(16)
  else { kh_set_error("paged_attn: head dim %d is not supported", hd); return -1; }
#undef LAUNCH_NARROW
#undef LAUNCH
#undef LAUNCH_W
  KH_LAUNCH_CHECK("paged_attn");
  return 0;
}

// ------------------------------------------------------------------------------- attention of prompt pieces
// Runs of consecutive positions of one sequence (prompts that join a step beside decoding sequences, short or chunked prompts):
// CTA = (up to 64 tokens, head), a warp per 16 tokens.  paged_attn_k spends about 14 instructions per token and key (unpacking,
// fp32 multiplies, shuffles): 6700 prompt tokens x 16 heads took 0.9 ms a layer.  Here the products run on the tensor
// cores (mma.sync: K and V rows come one by one through the block table), K and V tiles of 64 positions are copied once
// per CTA with cp.async, two in flight.  Nothing is rounded that was not before: q and k are bf16 in memory and their
// products accumulate in fp32; the probabilities stay fp32 and enter P V as three bf16 terms, whose 3 x 8 bits hold the 24
// of an fp32 mantissa.  The K order inside a 32-wide block is permuted identically for q and k so that fragments are whole
// 16-byte pieces.
constexpr int PP_ROWS = 64, PP_MAX_TILES = 1024;
struct PrefillTiles { int row0[PP_MAX_TILES]; uint8_t n[PP_MAX_TILES]; };

__device__ __forceinline__ void pp_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// x = hi + mid + lo, each bf16 (pairs packed)
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x, y);
  const float2 h = unpack_bf16(hi);
  mid = pack_bf16(x - h.x, y - h.y);
  const float2 m = unpack_bf16(mid);
  lo = pack_bf16(x - h.x - m.x, y - h.y - m.y);
}

// One token and head by one warp: positions 0..p of a cache at kc / vc (head offset included), output to dst.  The arithmetic of
// paged_attn_k, a key per lane group at a time.
template <int HD>
__device__ __noinline__ void attend_row(const bf16* q, const bf16* kc, const bf16* vc, const int* bt, int bs, int d, int p, float scale, bf16* dst) {
  constexpr int LPK = HD / 8, KPW = 32 / LPK;
  const int lane = threadIdx.x & 31, e0 = (lane % LPK) * 8;
  auto unpack8 = [](const uint4& u, float (&f)[8]) {
    const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), e = unpack_bf16(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = e.x; f[7] = e.y;
  };
  float x[8], k8[8], v8[8], o[8], m = -INFINITY, l = 0.f;
  unpack8(*reinterpret_cast<const uint4*>(q + e0), x);
#pragma unroll
  for (int i = 0; i < 8; i++) { x[i] *= scale; o[i] = 0.f; }
#pragma unroll 1
  for (int j0 = 0; j0 <= p; j0 += KPW) {
    const int j = j0 + lane / LPK, jj = min(j, p);
    const size_t at = ((size_t)__ldg(bt + jj / bs) * bs + jj % bs) * d + e0;
    unpack8(*reinterpret_cast<const uint4*>(kc + at), k8);
    unpack8(*reinterpret_cast<const uint4*>(vc + at), v8);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) s += k8[i] * x[i];
#pragma unroll
    for (int i = LPK / 2; i > 0; i >>= 1) s += __shfl_xor_sync(0xffffffffu, s, i);
    if (j <= p) {
      const float mn = fmaxf(m, s), ref = mn == -INFINITY ? 0.f : mn, sc = __expf(m - ref), pr = __expf(s - ref);
      m = mn;
      l = l * sc + pr;
#pragma unroll
      for (int i = 0; i < 8; i++) o[i] = o[i] * sc + pr * v8[i];
    }
  }
#pragma unroll
  for (int x2 = LPK; x2 < 32; x2 <<= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, x2), l2 = __shfl_xor_sync(0xffffffffu, l, x2);
    const float mn = fmaxf(m, m2), ref = mn == -INFINITY ? 0.f : mn, c1 = __expf(m - ref), c2 = __expf(m2 - ref);
    m = mn;
    l = l * c1 + l2 * c2;
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = o[i] * c1 + __shfl_xor_sync(0xffffffffu, o[i], x2) * c2;
  }
  const float inv = 1.f / l;
  if (lane < LPK)
    *reinterpret_cast<uint4*>(dst + e0) = make_uint4(pack_bf16(o[0] * inv, o[1] * inv), pack_bf16(o[2] * inv, o[3] * inv),
                                                     pack_bf16(o[4] * inv, o[5] * inv), pack_bf16(o[6] * inv, o[7] * inv));
}

template <int HD>
__global__ void __launch_bounds__(128)
paged_prefill_k(const __grid_constant__ PrefillTiles tiles, const bf16* __restrict__ qkv, int ld, const bf16* __restrict__ kc,
                const bf16* __restrict__ vc, bf16* __restrict__ out, const int* __restrict__ pos, const int* __restrict__ slot,
                const int* __restrict__ btab, int max_lb, int bs, int H, float scale, int max_ctx, int* err) {
  constexpr int PITCH = HD * 2 + 16, TILE = PP_ROWS * PITCH, PC = HD / 8;       // bytes per row, per tile; 16-byte pieces per row
  extern __shared__ __align__(16) uint8_t pp_smem[];                            // [2][K, V][64 rows]
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t base = smem_u32(pp_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c4 = lane & 3, h = blockIdx.y, d = H * HD;
  const int r0 = tiles.row0[blockIdx.x], p0 = pos[r0], sl = slot[r0];
  int n = tiles.n[blockIdx.x];
  // index guard as in paged_attn_k: tokens beyond the limits are recorded (status code 8) and skipped; they are the last of the run
  const int ok = sl < 0 || p0 < 0 ? 0 : min(n, min(max_ctx, max_lb * bs) - p0);
  if (ok < n && tid == 0) atomicCAS(err, 0, 8);
  if (ok <= 0) return;
  n = ok;
  const int ctx = p0 + n;
  const int* bt = btab + (size_t)sl * max_lb;
  auto load = [&](int kt) {                                                     // positions 64 kt .. into buffer kt & 1; zeros past the end
    const uint32_t dst = base + (kt & 1) * 2 * TILE;
#pragma unroll 4
    for (int i = tid; i < PP_ROWS * PC; i += 128) {
      const int r = i / PC, c = i % PC, j = kt * PP_ROWS + r;
      const int jb = j < ctx ? j / bs : 0;
      const size_t at = ((size_t)__ldg(bt + jb) * bs + (j < ctx ? j - jb * bs : 0)) * d + h * HD + c * 8;
      const uint32_t a = dst + r * PITCH + c * 16;
      const int bytes = j < ctx ? 16 : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(kc + at), "r"(bytes) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a + TILE), "l"(vc + at), "r"(bytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  const int w0 = warp * 16;                                                     // this warp's first token of the run
  uint4 q[HD / 32][2];                                                          // rows g and g + 8, piece c4 of every 32-wide block
#pragma unroll
  for (int j = 0; j < HD / 32; j++)
#pragma unroll
    for (int i = 0; i < 2; i++) {
      q[j][i] = make_uint4(0, 0, 0, 0);
      if (w0 + g + 8 * i < n) q[j][i] = *reinterpret_cast<const uint4*>(qkv + (size_t)(r0 + w0 + g + 8 * i) * ld + h * HD + j * 32 + c4 * 8);
    }
  float o[HD / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int t = 0; t < HD / 8; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[t][i] = 0.f;
  const int n_kt = (ctx + PP_ROWS - 1) / PP_ROWS;
#pragma unroll 1
  for (int kt = 0; kt < n_kt; kt++) {
    if (kt + 1 < n_kt) {
      load(kt + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int k0 = kt * PP_ROWS;
    if (w0 < n && k0 <= p0 + w0 + 15) {                                         // uniform over the warp
      const uint32_t sK = base + (kt & 1) * 2 * TILE, sV = sK + TILE;
      float s[8][4];
#pragma unroll
      for (int t = 0; t < 8; t++) {
#pragma unroll
        for (int i = 0; i < 4; i++) s[t][i] = 0.f;
#pragma unroll
        for (int j = 0; j < HD / 32; j++) {
          uint4 k;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(k.x), "=r"(k.y), "=r"(k.z), "=r"(k.w)
                       : "r"(sK + (t * 8 + g) * PITCH + j * 64 + c4 * 16) : "memory");
          pp_mma(s[t], q[j][0].x, q[j][1].x, q[j][0].y, q[j][1].y, k.x, k.y);
          pp_mma(s[t], q[j][0].z, q[j][1].z, q[j][0].w, q[j][1].w, k.z, k.w);
        }
      }
      float mx[2] = {m[0], m[1]};
#pragma unroll
      for (int t = 0; t < 8; t++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          s[t][i] *= scale;
          if (k0 + t * 8 + c4 * 2 + (i & 1) > p0 + w0 + g + 8 * (i >> 1)) s[t][i] = -INFINITY;
          mx[i >> 1] = fmaxf(mx[i >> 1], s[t][i]);
        }
      float ref[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        ref[i] = mx[i] == -INFINITY ? 0.f : mx[i];
        const float sc = __expf(m[i] - ref[i]);
        m[i] = mx[i];
        l[i] *= sc;
#pragma unroll
        for (int t = 0; t < HD / 8; t++) { o[t][2 * i] *= sc; o[t][2 * i + 1] *= sc; }
      }
#pragma unroll
      for (int t = 0; t < 8; t++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          s[t][i] = __expf(s[t][i] - ref[i >> 1]);
          l[i >> 1] += s[t][i];
        }
#pragma unroll
      for (int t = 0; t < 4; t++) {                                             // sixteen keys at a time
        uint32_t hi[4], mid[4], lo[4];
        split3(s[2 * t][0], s[2 * t][1], hi[0], mid[0], lo[0]);
        split3(s[2 * t][2], s[2 * t][3], hi[1], mid[1], lo[1]);
        split3(s[2 * t + 1][0], s[2 * t + 1][1], hi[2], mid[2], lo[2]);
        split3(s[2 * t + 1][2], s[2 * t + 1][3], hi[3], mid[3], lo[3]);
#pragma unroll
        for (int c = 0; c < HD; c += 16) {
          uint32_t b[4];
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                       : "r"(sV + (t * 16 + (lane & 15)) * PITCH + (c + (lane >> 4) * 8) * 2) : "memory");
          pp_mma(o[c / 8], hi[0], hi[1], hi[2], hi[3], b[0], b[1]);
          pp_mma(o[c / 8], mid[0], mid[1], mid[2], mid[3], b[0], b[1]);
          pp_mma(o[c / 8], lo[0], lo[1], lo[2], lo[3], b[0], b[1]);
          pp_mma(o[c / 8 + 1], hi[0], hi[1], hi[2], hi[3], b[2], b[3]);
          pp_mma(o[c / 8 + 1], mid[0], mid[1], mid[2], mid[3], b[2], b[3]);
          pp_mma(o[c / 8 + 1], lo[0], lo[1], lo[2], lo[3], b[2], b[3]);
        }
      }
    }
    __syncthreads();                                                            // the buffer is refilled in the next turn
  }
  // An infinity or NaN in V reaches the rows that see its position and no others.  The products above multiply it with the zeros of
  // masked positions and of the lower terms of P too, which leaves a NaN in every row of the warp: such a warp does its rows anew.
  uint32_t top = 0;
#pragma unroll
  for (int t = 0; t < HD / 8; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) top = max(top, __float_as_uint(o[t][i]) & 0x7fffffffu);
  if (__any_sync(0xffffffffu, top >= 0x7f800000u)) {
#pragma unroll 1
    for (int r = w0; r < min(n, w0 + 16); r++)
      attend_row<HD>(qkv + (size_t)(r0 + r) * ld + h * HD, kc + h * HD, vc + h * HD, bt, bs, d, p0 + r, scale,
                     out + (size_t)(r0 + r) * d + h * HD);
    return;
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    if (w0 + g + 8 * i < n) {
      const float inv = 1.f / l[i];
      bf16* dst = out + (size_t)(r0 + w0 + g + 8 * i) * d + h * HD + c4 * 2;
#pragma unroll
      for (int t = 0; t < HD / 8; t++) *reinterpret_cast<uint32_t*>(dst + t * 8) = pack_bf16(o[t][2 * i] * inv, o[t][2 * i + 1] * inv);
    }
  }
}
// Runs of tokens: `row0`, `len` (host arrays) give each run's first row in qkv / pos / slot / out and its length; the positions
// of a run are consecutive and belong to one sequence, and its K / V are in the cache already.
extern "C" int kh_paged_prefill(const void* qkv, int ld, const void* kc, const void* vc, void* out, const void* pos, const void* slot,
                                const void* btab, int max_lb, int bs, int H, int hd, float scale, int max_ctx, const void* row0,
                                const void* len, int n_runs, void* stream) {
  if (hd != 32 && hd != 64 && hd != 128) { kh_set_error("paged_prefill: head dim %d is not supported", hd); return -1; }
  if (((uintptr_t)qkv & 15) || ((uintptr_t)out & 15) || ((uintptr_t)kc & 15) || ((uintptr_t)vc & 15) || ld % 8) { kh_set_error("paged_prefill: misaligned operands"); return -1; }
  const int smem = 4 * PP_ROWS * (hd * 2 + 16);
  cudaStream_t st = (cudaStream_t)stream;
  PrefillTiles tiles;
  int nt = 0;
  auto flush = [&]() -> int {
    if (nt == 0) return 0;
#define LAUNCH(HD)                                                                                                              \
  {                                                                                                                             \
    if (smem > 48 * 1024 &&                                                                                                     \
        cudaFuncSetAttribute(paged_prefill_k<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {           \
      kh_set_error("paged_prefill: shared memory opt-in failed");                                                               \
      return -1;                                                                                                                \
    }                                                                                                                           \
    KH_LAUNCH((paged_prefill_k<HD>), dim3(nt, H), 128, smem, st, tiles, (const bf16*)qkv, ld, (const bf16*)kc, (const bf16*)vc,   \
              (bf16*)out, (const int*)pos, (const int*)slot, (const int*)btab, max_lb, bs, H, scale, max_ctx, kh_error_word_dev()); \
  }
    if (hd == 128) LAUNCH(128) else if (hd == 64) LAUNCH(64) else LAUNCH(32)
#undef LAUNCH
    KH_LAUNCH_CHECK("paged_prefill");
    nt = 0;
    return 0;
  };
  for (int i = 0; i < n_runs; i++) {
    const int r = ((const int*)row0)[i], n = ((const int*)len)[i];
    if (r < 0 || n < 1) { kh_set_error("paged_prefill: run %d is empty", i); return -1; }
    for (int at = (n - 1) / PP_ROWS * PP_ROWS; at >= 0; at -= PP_ROWS) {        // the pieces that see the most keys first
      tiles.row0[nt] = r + at;
      tiles.n[nt] = (uint8_t)(n - at < PP_ROWS ? n - at : PP_ROWS);
      if (++nt == PP_MAX_TILES && flush()) return -1;
    }
  }
  return flush();
}

// ------------------------------------------------------------------------------- split-KV attention
// Long contexts: the keys of a token are cut into `n_split` equal ranges, one CTA per (token, head,
// range) computes the softmax-weighted value sum over its range and its log-sum-exp, and a merge
// kernel combines the ranges (weights exp(lse_s - max lse)).  More CTAs per token than heads when a
// decode step has few sequences, and a score buffer of one range instead of the whole context.
// The range that holds position `pos` appends the token's k, v first (decode steps).
// Launched without programmatic dependence (KH_LAUNCH_AFTER): blocks that came while the GEMM before them still held the shared
// memory of part of the SMs all went to the others (4 layers of d2048, 32 sequences at 16300 positions: 5477 us a step, 3883 so).
template <int HD>
__global__ void __launch_bounds__(128)
paged_attn_split_k(const bf16* __restrict__ qkv, int ld, bf16* __restrict__ kc, bf16* __restrict__ vc,
                   float* __restrict__ o_part, float* __restrict__ lse_part, const int* __restrict__ pos,
                   const int* __restrict__ slot, const int* __restrict__ btab, int max_lb, int bs, int H, float scale,
                   int max_ctx, int chunk, int append, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y, sp = blockIdx.z, n_split = gridDim.z, tid = threadIdx.x;
  float* op = o_part + (((size_t)t * H + h) * n_split + sp) * HD;
  float* lp = lse_part + ((size_t)t * H + h) * n_split + sp;
  if (pos[t] < 0 || pos[t] >= max_ctx || pos[t] / bs >= max_lb || slot[t] < 0) {
    if (tid == 0) { atomicCAS(err, 0, 8); *lp = -INFINITY; }
    for (int e = tid; e < HD; e += 128) op[e] = 0.f;
    return;
  }
  extern __shared__ float sm[];
  constexpr int TPR = HD / 8, GROUPS = 128 / TPR;
  float* s_q = sm;
  float* s_p = sm + HD;              // `chunk` scores
  float* s_red = s_p + chunk;
  const int d = H * HD;
  const int ctx = pos[t] + 1;
  const int j0 = sp * chunk, j1 = min(ctx, j0 + chunk);
  const int* bt = btab + (size_t)slot[t] * max_lb;
  if (append && tid < 2 * TPR && ctx - 1 >= j0 && ctx - 1 < j1) {
    const int p = ctx - 1, which = tid / TPR, c = (tid % TPR) * 8;
    const size_t dst = ((size_t)bt[p / bs] * bs + (p % bs)) * d + h * HD + c;
    *reinterpret_cast<uint4*>((which ? vc : kc) + dst) =
        *reinterpret_cast<const uint4*>(qkv + (size_t)t * ld + (which + 1) * d + h * HD + c);
  }
  if (j1 <= j0) {                    // no keys in this range
    if (tid == 0) *lp = -INFINITY;
    for (int e = tid; e < HD; e += 128) op[e] = 0.f;
    return;
  }
  for (int e = tid; e < HD; e += 128) s_q[e] = __bfloat162float(qkv[(size_t)t * ld + h * HD + e]) * scale;
  __syncthreads();
  float lmax = -INFINITY;
  for (int j = j0 + tid; j < j1; j += 128) {
    const bf16* kp = kc + ((size_t)bt[j / bs] * bs + (j % bs)) * d + h * HD;
    float acc = 0.f;
#pragma unroll
    for (int c = 0; c < HD; c += 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(kp + c);
      const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), cc = unpack_bf16(v.z), e = unpack_bf16(v.w);
      acc += a.x * s_q[c] + a.y * s_q[c + 1] + b.x * s_q[c + 2] + b.y * s_q[c + 3] + cc.x * s_q[c + 4] +
             cc.y * s_q[c + 5] + e.x * s_q[c + 6] + e.y * s_q[c + 7];
    }
    s_p[j - j0] = acc;
    lmax = fmaxf(lmax, acc);
  }
  s_red[tid] = lmax;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if (tid < o) s_red[tid] = fmaxf(s_red[tid], s_red[tid + o]);
    __syncthreads();
  }
  const float gmax = s_red[0];
  __syncthreads();
  float lsum = 0.f;
  for (int j = j0 + tid; j < j1; j += 128) {
    const float e = __expf(s_p[j - j0] - gmax);
    s_p[j - j0] = e;
    lsum += e;
  }
  s_red[tid] = lsum;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if (tid < o) s_red[tid] += s_red[tid + o];
    __syncthreads();
  }
  const float tot = s_red[0];
  __syncthreads();
  const int c8 = (tid % TPR) * 8, grp = tid / TPR;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; k++) acc[k] = 0.f;
  for (int j = j0 + grp; j < j1; j += GROUPS) {
    const uint4 v = *reinterpret_cast<const uint4*>(vc + ((size_t)bt[j / bs] * bs + (j % bs)) * d + h * HD + c8);
    const float pj = s_p[j - j0];
    const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), cc = unpack_bf16(v.z), e = unpack_bf16(v.w);
    acc[0] += pj * a.x; acc[1] += pj * a.y; acc[2] += pj * b.x; acc[3] += pj * b.y;
    acc[4] += pj * cc.x; acc[5] += pj * cc.y; acc[6] += pj * e.x; acc[7] += pj * e.y;
  }
#pragma unroll
  for (int k = 0; k < 8; k++) s_red[grp * HD + c8 + k] = acc[k];
  __syncthreads();
  if (tid < HD) {
    float o = 0.f;
    for (int g = 0; g < GROUPS; g++) o += s_red[g * HD + tid];
    op[tid] = o / tot;
  }
  if (tid == 0) *lp = gmax + logf(tot);
}
// out[t, h, :] = sum_s w_s o_part[t, h, s, :] / sum_s w_s with w_s = exp(lse_s - max_s lse_s), ranges in index order
__global__ void paged_attn_merge_k(const float* __restrict__ o_part, const float* __restrict__ lse_part, bf16* __restrict__ out,
                                   int H, int HD, int n_split) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y, e = threadIdx.x;
  const float* lp = lse_part + ((size_t)t * H + h) * n_split;
  float m = -INFINITY;
  for (int s = 0; s < n_split; s++) m = fmaxf(m, lp[s]);
  float num = 0.f, den = 0.f;
  if (m > -INFINITY)
    for (int s = 0; s < n_split; s++) {
      const float w = lp[s] == -INFINITY ? 0.f : __expf(lp[s] - m);
      num += w * o_part[(((size_t)t * H + h) * n_split + s) * HD + e];
      den += w;
    }
  out[((size_t)t * H + h) * HD + e] = __float2bfloat16(den > 0.f ? num / den : 0.f);
}
// `o_part`: ntok * H * n_split * hd floats, `lse_part`: ntok * H * n_split floats (scratch).
extern "C" int kh_paged_attn_split(const void* qkv, int ld, void* kc, void* vc, void* out, void* o_part, void* lse_part,
                                   const void* pos, const void* slot, const void* btab, int max_lb, int bs, int H, int hd,
                                   float scale, int ntok, int max_ctx, int n_split, int append, void* stream) {
  if (n_split < 1 || n_split > 64) { kh_set_error("paged_attn_split: n_split %d out of range", n_split); return -1; }
  const int chunk = (max_ctx + n_split - 1) / n_split;
  const size_t smem = (size_t)(hd + chunk + 1024 + 8) * sizeof(float);
  if (smem > 200 * 1024) { kh_set_error("paged_attn_split: a range of %d positions does not fit in shared memory", chunk); return -1; }
  dim3 grid(ntok, H, n_split);
  cudaStream_t st = (cudaStream_t)stream;
#define LAUNCH(HD)                                                                                                        \
  {                                                                                                                       \
    static size_t attr = 48 * 1024;                                                                                       \
    if (smem > attr) { cudaFuncSetAttribute(paged_attn_split_k<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); attr = smem; } \
    KH_LAUNCH_AFTER((paged_attn_split_k<HD>), grid, 128, smem, st, (const bf16*)qkv, ld, (bf16*)kc, (bf16*)vc, (float*)o_part,  \
              (float*)lse_part, (const int*)pos, (const int*)slot, (const int*)btab, max_lb, bs, H, scale, max_ctx, chunk, \
              append, kh_error_word_dev());                                                                               \
  }
  if (hd == 128) LAUNCH(128)
  else if (hd == 64) LAUNCH(64)
  else if (hd == 32) LAUNCH(32)
  else if (hd == 16) LAUNCH(16)
  else { kh_set_error("paged_attn_split: head dim %d is not supported", hd); return -1; }
#undef LAUNCH
  KH_LAUNCH_CHECK("paged_attn_split");
  KH_LAUNCH(paged_attn_merge_k, dim3(ntok, H), hd, 0, st, (const float*)o_part, (const float*)lse_part, (bf16*)out, H, hd, n_split);
  KH_LAUNCH_CHECK("paged_attn_merge");
  return 0;
}

// ------------------------------------------------------------------------------- gather / copy
__global__ void gather_rows_k(const bf16* __restrict__ x, const int* __restrict__ rows, bf16* __restrict__ out, int d) {
  pdl_wait();
  pdl_launch_dependents();
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)rows[blockIdx.x] * d);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.x * d);
  for (int i = threadIdx.x; i < d / 8; i += blockDim.x) dst[i] = src[i];
}
extern "C" int kh_gather_rows(const void* x, const void* rows, void* out, int nseq, int d, void* stream) {
  if (d % 8) { kh_set_error("gather_rows: d must be a multiple of 8"); return -1; }
  KH_LAUNCH(gather_rows_k, nseq, 128, 0, (cudaStream_t)stream, (const bf16*)x, (const int*)rows, (bf16*)out, d);
  KH_LAUNCH_CHECK("gather_rows");
  return 0;
}
// Copies whole KV blocks (src -> dst pairs) in every layer: the device half of copy-on-write.
__global__ void copy_blocks_k(bf16* __restrict__ kc, bf16* __restrict__ vc, const int* __restrict__ pairs,
                              size_t block_elems, size_t layer_elems) {
  pdl_wait();
  pdl_launch_dependents();
  const int pr = blockIdx.x, layer = blockIdx.y;
  const size_t src = (size_t)layer * layer_elems + (size_t)pairs[2 * pr] * block_elems;
  const size_t dst = (size_t)layer * layer_elems + (size_t)pairs[2 * pr + 1] * block_elems;
  for (size_t i = threadIdx.x * 8; i < block_elems; i += blockDim.x * 8) {
    *reinterpret_cast<uint4*>(kc + dst + i) = *reinterpret_cast<const uint4*>(kc + src + i);
    *reinterpret_cast<uint4*>(vc + dst + i) = *reinterpret_cast<const uint4*>(vc + src + i);
  }
}
extern "C" int kh_copy_blocks(void* kc, void* vc, const void* pairs, int npairs, int n_layer, long block_elems,
                              long layer_elems, void* stream) {
  if (npairs <= 0) return 0;
  if (block_elems % 8) { kh_set_error("copy_blocks: block size must be a multiple of 8 elements"); return -1; }
  dim3 grid(npairs, n_layer);
  KH_LAUNCH(copy_blocks_k, grid, 128, 0, (cudaStream_t)stream, (bf16*)kc, (bf16*)vc, (const int*)pairs, (size_t)block_elems,
                                                        (size_t)layer_elems);
  KH_LAUNCH_CHECK("copy_blocks");
  return 0;
}

// ------------------------------------------------------------------------------- sampler
// One CTA per sequence.  temperature <= 0: argmax (lowest index wins ties).  Otherwise a draw
// from softmax(logits / temperature): each thread owns a contiguous chunk, chunk sums are
// scanned in order, the draw u * total picks the chunk and then the element -- deterministic
// for a given (seed, step, row).  `rep` > 1 draws `rep` independent tokens from the same row
// (first token of a forked group).
__device__ __forceinline__ uint32_t mix32(uint64_t x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdULL; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ULL; x ^= x >> 33;
  return (uint32_t)(x >> 16);
}
__global__ void __launch_bounds__(256)
sample_k(const bf16* __restrict__ logits, int ld, int V, float temperature, unsigned long long seed, int step,
         const int* __restrict__ step_dev, int rep, int* __restrict__ out) {
  pdl_wait();
  pdl_launch_dependents();
  if (step_dev) {      // step number and seed kept in device memory: a captured launch draws fresh numbers
    step = step_dev[0];
    seed = (unsigned long long)(unsigned)step_dev[1] | ((unsigned long long)(unsigned)step_dev[2] << 32);
  }
  __shared__ float s_v[256];
  __shared__ int s_i[256];
  __shared__ float s_scan[257];
  const int row = blockIdx.x, tid = threadIdx.x;
  const bf16* lg = logits + (size_t)row * ld;
  const int chunk = (V + 255) / 256;
  const int c0 = tid * chunk, c1 = min(V, c0 + chunk);
  float best = -INFINITY;
  int bi = V;
  for (int i = c0; i < c1; i++) {
    float x = __bfloat162float(lg[i]);
    if (x > best) { best = x; bi = i; }
  }
  s_v[tid] = best; s_i[tid] = bi;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o) {
      float a = s_v[tid], b = s_v[tid + o];
      int ia = s_i[tid], ib = s_i[tid + o];
      if (b > a || (b == a && ib < ia)) { s_v[tid] = b; s_i[tid] = ib; }
    }
    __syncthreads();
  }
  const float gmax = s_v[0];
  const int gidx = s_i[0];
  if (temperature <= 0.f) {
    if (tid < rep) out[row * rep + tid] = gidx;
    return;
  }
  const float it = 1.f / temperature;
  float sum = 0.f;
  for (int i = c0; i < c1; i++) sum += __expf((__bfloat162float(lg[i]) - gmax) * it);
  __syncthreads();
  s_scan[tid + 1] = sum;
  if (tid == 0) s_scan[0] = 0.f;
  __syncthreads();
  if (tid == 0) for (int k = 1; k <= 256; k++) s_scan[k] += s_scan[k - 1];   // ordered, 256 adds
  __syncthreads();
  const float total = s_scan[256];
  for (int r = 0; r < rep; r++) {
    const uint32_t rnd = mix32(seed * 0x9E3779B97F4A7C15ULL + (uint64_t)step * 1000003ULL + (uint64_t)(row * rep + r) * 7919ULL);
    const float u = ((rnd >> 8) + 0.5f) * (1.f / 16777216.f) * total;
    if (u >= s_scan[tid] && (u < s_scan[tid + 1] || (tid == 255))) {
      float acc = s_scan[tid];
      int pick = max(c0, min(c1, V) - 1);
      for (int i = c0; i < c1; i++) {
        acc += __expf((__bfloat162float(lg[i]) - gmax) * it);
        if (u < acc) { pick = i; break; }
      }
      if (c0 >= V) pick = gidx;
      out[row * rep + r] = pick;
    }
  }
}
// Greedy rows: the same argmax (lowest index wins ties, NaN never wins) with 16-byte loads, eight in flight a thread, and 1024 or
// 256 threads.  sample_k's contiguous chunks per thread, which the draw needs, read 2 bytes at a time.  us for 1 / 512 rows, sample_k /
// 1024 / 256 threads: V = 2049 2.6 / 2.2 / 2.0 and 3.3 / 7.3 / 2.6, V = 8000 4.2 / 2.1 / 1.9 and 10.8 / 7.2 / 3.4,
// V = 50257 13.2 / 3.4 / 4.4 and 46.8 / 12.6 / 9.8.
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
argmax_k(const bf16* __restrict__ logits, int ld, int V, int rep, int* __restrict__ out) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int WARPS = THREADS / 32;
  __shared__ float s_v[WARPS];
  __shared__ int s_i[WARPS];
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const bf16* lg = logits + (size_t)row * ld;
  float best = -INFINITY;
  int bi = V;
  auto take = [&](float x, int i) { if (x > best) { best = x; bi = i; } };       // indices rise within a thread
  const int nv = ((uintptr_t)lg & 15) == 0 ? V / 8 : 0;                           // whole 16-byte pieces
  for (int c0 = tid; c0 < nv; c0 += 8 * THREADS) {
    uint4 u[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (c0 + k * THREADS < nv) u[k] = __ldg(reinterpret_cast<const uint4*>(lg) + c0 + k * THREADS);
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (c0 + k * THREADS < nv) {
        const int i = (c0 + k * THREADS) * 8;
        const float2 a = unpack_bf16(u[k].x), b = unpack_bf16(u[k].y), c = unpack_bf16(u[k].z), e = unpack_bf16(u[k].w);
        take(a.x, i); take(a.y, i + 1); take(b.x, i + 2); take(b.y, i + 3);
        take(c.x, i + 4); take(c.y, i + 5); take(e.x, i + 6); take(e.y, i + 7);
      }
  }
  for (int i = nv * 8 + tid; i < V; i += THREADS) take(__bfloat162float(lg[i]), i);
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float b = __shfl_xor_sync(0xffffffffu, best, o);
      const int ib = __shfl_xor_sync(0xffffffffu, bi, o);
      if (b > best || (b == best && ib < bi)) { best = b; bi = ib; }
    }
  };
  reduce();
  if (lane == 0) { s_v[tid >> 5] = best; s_i[tid >> 5] = bi; }
  __syncthreads();
  if (tid >= 32) return;
  best = lane < WARPS ? s_v[lane] : -INFINITY;
  bi = lane < WARPS ? s_i[lane] : V;
  reduce();
  for (int r = lane; r < rep; r += 32) out[row * rep + r] = bi;
}
// `step_dev` (optional): three device words {step number, seed low, seed high}; when given they replace
// `step` and `seed`, so that the launch can be replayed from a CUDA graph with new values each time.
extern "C" int kh_sample2(const void* logits, int ld, int V, float temperature, unsigned long long seed, int step,
                          const void* step_dev, int rep, void* out, int nseq, void* stream) {
  if (rep < 1 || rep > 256) { kh_set_error("sample: rep must be in [1, 256]"); return -1; }
  if (temperature <= 0.f && V > 2048) {
    // one turn of loads takes up to 16384 logits with 256 threads; more rows than SMs share an SM, where a CTA of 1024 threads
    // costs more than it loads
    if (V > 16384 && nseq <= 148) KH_LAUNCH(argmax_k<1024>, nseq, 1024, 0, (cudaStream_t)stream, (const bf16*)logits, ld, V, rep, (int*)out);
    else KH_LAUNCH(argmax_k<256>, nseq, 256, 0, (cudaStream_t)stream, (const bf16*)logits, ld, V, rep, (int*)out);
    KH_LAUNCH_CHECK("sample");
    return 0;
  }
  KH_LAUNCH(sample_k, nseq, 256, 0, (cudaStream_t)stream, (const bf16*)logits, ld, V, temperature, seed, step,
            (const int*)step_dev, rep, (int*)out);
  KH_LAUNCH_CHECK("sample");
  return 0;
}
extern "C" int kh_sample(const void* logits, int ld, int V, float temperature, unsigned long long seed, int step,
                         int rep, void* out, int nseq, void* stream) {
  return kh_sample2(logits, ld, V, temperature, seed, step, nullptr, rep, out, nseq, stream);
}
