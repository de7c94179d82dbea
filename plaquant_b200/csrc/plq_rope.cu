// Rotary position embedding of the query and key heads of a fused QKV projection and the append of the keys and
// values to the cache, in one pass over the projection's output (inference/forward_pass.py:82-110 and 216-247 in
// the reference: apply_rotary_pos_emb, then the cache update).  HBM-bound: every element of [rows, (h + 2 kv) * 128]
// is read once and written once.
//
// Arithmetic, per element pair (x1 = element i of the head's first half, x2 = element i of its second half), in
// float32 with every operation rounded on its own (no fused multiply-add), then one rounding to bf16:
//     out[i]      = x1 * cos[i]      + (-x2) * sin[i]
//     out[64 + i] = x2 * cos[64 + i] +   x1  * sin[64 + i]
// which is `x.float() * cos + rotate_half(x).float() * sin` of the PyTorch formulation, bit for bit.
#include "plq_common.cuh"
#include "plq_quant.cuh"

namespace plq {

constexpr int kRopeHeadDim = 128;

// Packed rows of keys and values -> their bf16 values.
struct UnpackRowsArgs {
  const uint8_t* src[2];     // [batch, t_max, kv_heads, 72]
  uint4* dst[2];             // bf16 [batch, t, kv_heads, 128]
  long long t_heads, cap_heads, total;     // t * kv_heads, t_max * kv_heads, threads per cache = batch * t * kv_heads * 16
  int kv_heads;
};

struct RopeArgs {
  const uint4* qkv;        // bf16 [rows, ld]: [q heads | k heads | v heads] per row
  const float* cos;        // float32 [t, 128]: row tt belongs to position pos + tt
  const float* sin;
  uint4* q_out;            // bf16 [rows, heads, 128]
  uint4* k_dst;            // bf16 [batch, t_max, kv_heads, 128]
  uint4* v_dst;
  const long long* pos_dev;  // device scalar: first cache position of this call, or nullptr to use `pos`
  long long pos, t_max;
  int* status;
  long long ld8;           // row stride of qkv in 16-byte units
  long long total;         // rows * (heads + 2 kv_heads) * 8 threads
  int t, heads, kv_heads;
  // packed cache only
  UnpackRowsArgs old;      // the caches' bf16 values, or dst = nullptr
  float2* q_f32;           // the queries as float32 (bf16-valued) instead of q_out
  long long ctx;           // positions of `old`
  unsigned append_blocks;
};

__device__ __forceinline__ void unpack_bf16x8(const uint4& q, float (&f)[8]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Programmatic dependent launch on both sides, like the pack kernels: a few microseconds of work in a decode step, of
// which the launch latency would be a third.
__global__ void __launch_bounds__(256, 6) rope_kv_append_kernel(const RopeArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= a.total) return;
  const int all_heads = a.heads + 2 * a.kv_heads;
  const int j = static_cast<int>(idx & 7);                              // which 8 elements of each half
  const int head = static_cast<int>((idx >> 3) % all_heads);
  const long long row = (idx >> 3) / all_heads;
  const long long b = row / a.t;
  const int tt = static_cast<int>(row - b * a.t);
  const uint4* src = a.qkv + row * a.ld8 + static_cast<long long>(head) * 16 + j;
  uint4 lo = src[0], hi = src[8];
  if (head < a.heads + a.kv_heads) {
    float x1[8], x2[8];
    unpack_bf16x8(lo, x1);
    unpack_bf16x8(hi, x2);
    const float4* c1 = reinterpret_cast<const float4*>(a.cos + static_cast<size_t>(tt) * kRopeHeadDim + 8 * j);
    const float4* s1 = reinterpret_cast<const float4*>(a.sin + static_cast<size_t>(tt) * kRopeHeadDim + 8 * j);
    const float4 ca = c1[0], cb = c1[1], cc = c1[16], cd = c1[17];      // cos[8j..8j+7], cos[64+8j..]
    const float4 sa = s1[0], sb = s1[1], sc = s1[16], sd = s1[17];
    const float cl[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    const float ch[8] = {cc.x, cc.y, cc.z, cc.w, cd.x, cd.y, cd.z, cd.w};
    const float sl[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
    const float sh[8] = {sc.x, sc.y, sc.z, sc.w, sd.x, sd.y, sd.z, sd.w};
    float o1[8], o2[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o1[i] = __fadd_rn(__fmul_rn(x1[i], cl[i]), __fmul_rn(-x2[i], sl[i]));
      o2[i] = __fadd_rn(__fmul_rn(x2[i], ch[i]), __fmul_rn(x1[i], sh[i]));
    }
    lo = make_uint4(pack_bf16x2(o1[0], o1[1]), pack_bf16x2(o1[2], o1[3]), pack_bf16x2(o1[4], o1[5]), pack_bf16x2(o1[6], o1[7]));
    hi = make_uint4(pack_bf16x2(o2[0], o2[1]), pack_bf16x2(o2[2], o2[3]), pack_bf16x2(o2[4], o2[5]), pack_bf16x2(o2[6], o2[7]));
  }
  uint4* dst;
  if (head < a.heads) {
    dst = a.q_out + (row * a.heads + head) * 16 + j;
  } else {
    const long long p = (a.pos_dev != nullptr ? *a.pos_dev : a.pos) + tt;
    if (p < 0 || p >= a.t_max) {                     // the cache is full: nothing is stored, the caller is told
      if (a.status != nullptr) atomicExch(a.status, PLQ_DEV_RANGE);
      return;
    }
    const bool is_k = head < a.heads + a.kv_heads;
    const int kh = head - a.heads - (is_k ? 0 : a.kv_heads);
    dst = (is_k ? a.k_dst : a.v_dst) + ((b * a.t_max + p) * a.kv_heads + kh) * 16 + j;
  }
  dst[0] = lo;
  dst[8] = hi;
}

// ---- the same with a packed cache ------------------------------------------------------------------------------
// Rows of the NVFP4 cache: 64 bytes of E2M1 codes, 8 E4M3 scale bytes.  One warp per head row, lane l holding elements
// (2 l, 2 l + 1) and (64 + 2 l, 65 + 2 l): RoPE and the last butterfly stage stay in the lane, a 16-element block is
// eight lanes.  Replaces, per decode step and layer, fifteen elementwise, pack and concatenation launches over a few
// hundred rows each; those were bound by their launches.
constexpr int kPackedRow = 72;

struct HeadRow { float2 a, b; };

__device__ __forceinline__ HeadRow bf16_row(float2 a, float2 b) {
  const uint32_t w0 = f32x2_to_bf16x2(a.x, a.y), w1 = f32x2_to_bf16x2(b.x, b.y);
  return {make_float2(bf16lo_to_f32(w0), bf16hi_to_f32(w0)), make_float2(bf16lo_to_f32(w1), bf16hi_to_f32(w1))};
}
__device__ __forceinline__ HeadRow rope_row(const HeadRow& x, const float* cos, const float* sin, int lane) {
  const float2 c1 = *reinterpret_cast<const float2*>(cos + 2 * lane), c2 = *reinterpret_cast<const float2*>(cos + 64 + 2 * lane);
  const float2 s1 = *reinterpret_cast<const float2*>(sin + 2 * lane), s2 = *reinterpret_cast<const float2*>(sin + 64 + 2 * lane);
  float2 lo, hi;
  lo.x = __fadd_rn(__fmul_rn(x.a.x, c1.x), __fmul_rn(-x.b.x, s1.x));
  lo.y = __fadd_rn(__fmul_rn(x.a.y, c1.y), __fmul_rn(-x.b.y, s1.y));
  hi.x = __fadd_rn(__fmul_rn(x.b.x, c2.x), __fmul_rn(x.a.x, s2.x));
  hi.y = __fadd_rn(__fmul_rn(x.b.y, c2.y), __fmul_rn(x.a.y, s2.y));
  return bf16_row(lo, hi);
}
// Block-Hadamard(128), stages of stride 1, 2, .. 64 in this order and one rounding to bf16: bit for bit the rotation
// of the pack kernels (up to the sign of a zero, which the quantiser drops).
__device__ __forceinline__ HeadRow hadamard_row(HeadRow x, int lane) {
  x.a = make_float2(__fadd_rn(x.a.x, x.a.y), __fsub_rn(x.a.x, x.a.y));
  x.b = make_float2(__fadd_rn(x.b.x, x.b.y), __fsub_rn(x.b.x, x.b.y));
#pragma unroll
  for (int h = 1; h < 32; h <<= 1) {
    const bool up = (lane & h) != 0;               // this lane holds the upper element: partner - own
    float* e[4] = {&x.a.x, &x.a.y, &x.b.x, &x.b.y};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float o = __shfl_xor_sync(0xFFFFFFFFu, *e[i], h);
      *e[i] = up ? __fsub_rn(o, *e[i]) : __fadd_rn(*e[i], o);
    }
  }
  const float c = 0.088388347648318441f;           // 1/sqrt(128)
  return bf16_row(make_float2(__fmul_rn(__fadd_rn(x.a.x, x.b.x), c), __fmul_rn(__fadd_rn(x.a.y, x.b.y), c)),
                  make_float2(__fmul_rn(__fsub_rn(x.a.x, x.b.x), c), __fmul_rn(__fsub_rn(x.a.y, x.b.y), c)));
}
// The value of one E2M1 code.  Times its E4M3 scale it has at most 6 significant bits: exact in bf16.
__device__ __forceinline__ float e2m1_value(uint32_t c) {
  const uint32_t mag = c & 7;
  const float mv = mag < 2 ? 0.5f * mag : __uint_as_float(((mag >> 1) + 126u) << 23 | (mag & 1u) << 22);
  return (c & 8) ? -mv : mv;
}

// Quantises the row into the cache and, where `values` is given, leaves there what the cache now holds.
__device__ __forceinline__ void store_nvfp4_row(uint8_t* p, uint32_t* values, const HeadRow& x, int lane) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const float2 v = half ? x.b : x.a;
    float m = fmaxf(fabsf(v.x), fabsf(v.y));
    m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
    m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 4));
    const uint32_t c = nvfp4_scale_code(m);
    const float s = e4m3_code_to_f32(c);
    const uint32_t code = nvfp4_quantize2(v, rcp_approx(s));
    p[32 * half + lane] = static_cast<uint8_t>(code);
    if (values != nullptr) values[32 * half + lane] = pack_bf16x2(e2m1_value(code & 0xF) * s, e2m1_value(code >> 4) * s);
    if ((lane & 7) == 0) p[64 + 4 * half + (lane >> 3)] = static_cast<uint8_t>(c);
  }
}

// Packed rows of keys and values -> bf16, both caches, straight out of allocations with room for t_max positions: eight
// elements (four code bytes, one scale byte) per thread, 16-byte stores.  Bound by the bytes written (256 per 72 read).
// The positions [skip, skip + n_skip) are left to whoever appends them.
__device__ __forceinline__ void unpack_rows(const UnpackRowsArgs& a, long long block, long long skip, int n_skip) {
  const long long i = block * blockDim.x + threadIdx.x;
  if (i >= 2 * a.total) return;
  const bool value = i >= a.total;
  const long long idx = value ? i - a.total : i;
  const long long r = idx >> 4, b = r / a.t_heads, in_seq = r - b * a.t_heads;
  if (n_skip != 0) {
    const long long p = in_seq / a.kv_heads;
    if (p >= skip && p < skip + n_skip) return;
  }
  const int j = static_cast<int>(idx & 15);
  const uint8_t* p = (value ? a.src[1] : a.src[0]) + (b * a.cap_heads + in_seq) * kPackedRow;
  const uint32_t codes = *reinterpret_cast<const uint32_t*>(p + 4 * j);
  const float s = e4m3_code_to_f32(p[64 + (j >> 1)]);
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = pack_bf16x2(e2m1_value(codes >> (8 * k) & 0xF) * s, e2m1_value(codes >> (8 * k + 4) & 0xF) * s);
  (value ? a.dst[1] : a.dst[0])[idx] = make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(256) unpack_head_rows_kernel(const UnpackRowsArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  unpack_rows(a, blockIdx.x, 0, 0);
}

// One launch for a step over a packed cache: the first blocks rotate and append (and leave the new rows' values beside
// the old ones'), the others dequantise the rows that were there.  As three launches - append, dequantisation, the
// queries' widening to float32 - a decode step spent most of them waiting for the launch before.
__global__ void __launch_bounds__(256) rope_kv_append_nvfp4_kernel(const RopeArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  if (blockIdx.x >= a.append_blocks) {             // the rows that were in the cache before
    unpack_rows(a.old, blockIdx.x - a.append_blocks, (a.pos_dev != nullptr ? *a.pos_dev : a.pos), a.t);
    return;
  }
  const long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;      // head row
  if (idx >= a.total) return;
  const int lane = threadIdx.x & 31;
  const int all_heads = a.heads + 2 * a.kv_heads;
  const int head = static_cast<int>(idx % all_heads);
  const long long row = idx / all_heads;
  const long long b = row / a.t;
  const int tt = static_cast<int>(row - b * a.t);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(a.qkv + row * a.ld8 + static_cast<long long>(head) * 16) + lane;
  const uint32_t w0 = src[0], w1 = src[32];
  HeadRow x = {make_float2(bf16lo_to_f32(w0), bf16hi_to_f32(w0)), make_float2(bf16lo_to_f32(w1), bf16hi_to_f32(w1))};
  const bool is_q = head < a.heads, is_k = !is_q && head < a.heads + a.kv_heads;
  if (is_q || is_k) x = rope_row(x, a.cos + static_cast<size_t>(tt) * kRopeHeadDim, a.sin + static_cast<size_t>(tt) * kRopeHeadDim, lane);
  if (is_q && a.q_f32 != nullptr) {
    float2* dst = a.q_f32 + (row * a.heads + head) * 64 + lane;
    dst[0] = x.a;
    dst[32] = x.b;
    return;
  }
  if (is_q) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(a.q_out + (row * a.heads + head) * 16) + lane;
    dst[0] = f32x2_to_bf16x2(x.a.x, x.a.y);
    dst[32] = f32x2_to_bf16x2(x.b.x, x.b.y);
    return;
  }
  const long long p = (a.pos_dev != nullptr ? *a.pos_dev : a.pos) + tt;
  if (p < 0 || p >= a.t_max) {                       // the cache is full: nothing is stored, the caller is told
    if (lane == 0 && a.status != nullptr) atomicExch(a.status, PLQ_DEV_RANGE);
    return;
  }
  if (is_k) x = hadamard_row(x, lane);
  const int kh = head - a.heads - (is_k ? 0 : a.kv_heads);
  uint4* values = is_k ? a.old.dst[0] : a.old.dst[1];
  if (p >= a.ctx) values = nullptr;
  if (values != nullptr) values += ((b * a.ctx + p) * a.kv_heads + kh) * 16;
  store_nvfp4_row(reinterpret_cast<uint8_t*>(is_k ? a.k_dst : a.v_dst) + ((b * a.t_max + p) * a.kv_heads + kh) * kPackedRow,
                  reinterpret_cast<uint32_t*>(values), x, lane);
}

template <typename Args>
static int launch_overlapped(void (*kernel)(const Args), dim3 grid, const Args& a, void* stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PLQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, a));
  return PLQ_OK;
}

static UnpackRowsArgs unpack_args(const void* k_rows, const void* v_rows, int64_t batch, int64_t t, int64_t t_max, int64_t kv_heads,
                                  void* k_bf16, void* v_bf16) {
  UnpackRowsArgs a;
  a.src[0] = static_cast<const uint8_t*>(k_rows);
  a.src[1] = static_cast<const uint8_t*>(v_rows);
  a.dst[0] = static_cast<uint4*>(k_bf16);
  a.dst[1] = static_cast<uint4*>(v_bf16);
  a.t_heads = t * kv_heads;
  a.cap_heads = t_max * kv_heads;
  a.total = batch * t * kv_heads * 16;
  a.kv_heads = static_cast<int>(kv_heads);
  return a;
}

// With `ctx` (packed cache): q_out is float32, and k_values / v_values receive the first ctx positions.
static int launch_rope(bool packed, const void* qkv_bf16, int64_t ld, const void* cos_f32, const void* sin_f32,
                       int64_t batch, int64_t t, int64_t heads, int64_t kv_heads, int64_t head_dim,
                       void* q_out_bf16, void* k_cache, void* v_cache, int64_t t_max,
                       const int64_t* pos_dev, int64_t pos, int32_t* dev_status, void* stream, int64_t ctx = 0,
                       void* k_values = nullptr, void* v_values = nullptr) {
  if (head_dim != kRopeHeadDim) return PLQ_ERR_SHAPE;
  if (batch < 1 || t < 1 || heads < 1 || kv_heads < 1 || t_max < 1) return PLQ_ERR_SHAPE;
  if (ld < (heads + 2 * kv_heads) * kRopeHeadDim || ld % 8 != 0) return PLQ_ERR_SHAPE;
  if (pos_dev == nullptr && (pos < 0 || pos + t > t_max)) return PLQ_ERR_SHAPE;
  if (batch * t > 0x7FFFFFFF || heads + 2 * kv_heads > 4096) return PLQ_ERR_LIMIT;
  if (!qkv_bf16 || !cos_f32 || !sin_f32 || !q_out_bf16 || !k_cache || !v_cache) return PLQ_ERR_NULL;
  if (!aligned16(qkv_bf16) || !aligned16(cos_f32) || !aligned16(sin_f32) || !aligned16(q_out_bf16) ||
      !aligned16(k_cache) || !aligned16(v_cache))
    return PLQ_ERR_ALIGN;
  int st = device_check();
  if (st != PLQ_OK) return st;
  RopeArgs a;
  a.qkv = static_cast<const uint4*>(qkv_bf16);
  a.cos = static_cast<const float*>(cos_f32);
  a.sin = static_cast<const float*>(sin_f32);
  a.q_out = static_cast<uint4*>(q_out_bf16);
  a.k_dst = static_cast<uint4*>(k_cache);
  a.v_dst = static_cast<uint4*>(v_cache);
  a.pos_dev = reinterpret_cast<const long long*>(pos_dev);
  a.pos = pos;
  a.t_max = t_max;
  a.status = dev_status;
  a.ld8 = ld / 8;
  a.total = batch * t * (heads + 2 * kv_heads) * (packed ? 1 : 8);      // head rows, or threads
  a.t = static_cast<int>(t);
  a.heads = static_cast<int>(heads);
  a.kv_heads = static_cast<int>(kv_heads);
  a.old = unpack_args(k_cache, v_cache, batch, ctx, t_max, kv_heads, k_values, v_values);
  a.q_f32 = ctx > 0 ? static_cast<float2*>(q_out_bf16) : nullptr;
  a.ctx = ctx;
  a.append_blocks = static_cast<unsigned>((a.total + 7) / 8);
  if (packed) {
    // positions that are appended need no block of their own; a prompt has no others
    const long long blocks = a.append_blocks + (ctx > t || (ctx > 0 && pos_dev) ? (2 * a.old.total + 255) / 256 : 0);
    if (blocks > 0x7FFFFFFF) return PLQ_ERR_LIMIT;
    return launch_overlapped(rope_kv_append_nvfp4_kernel, dim3(static_cast<unsigned>(blocks)), a, stream);
  }
  return launch_overlapped(rope_kv_append_kernel, dim3(static_cast<unsigned>((a.total + 255) / 256)), a, stream);
}

}  // namespace plq

extern "C" int plq_rope_kv_append(const void* qkv_bf16, int64_t ld, const void* cos_f32, const void* sin_f32,
                                  int64_t batch, int64_t t, int64_t heads, int64_t kv_heads, int64_t head_dim,
                                  void* q_out_bf16, void* k_cache_bf16, void* v_cache_bf16, int64_t t_max,
                                  const int64_t* pos_dev, int64_t pos, int32_t* dev_status, void* stream) {
  return plq::launch_rope(false, qkv_bf16, ld, cos_f32, sin_f32, batch, t, heads, kv_heads, head_dim, q_out_bf16, k_cache_bf16,
                          v_cache_bf16, t_max, pos_dev, pos, dev_status, stream);
}

extern "C" int plq_rope_kv_append_nvfp4(const void* qkv_bf16, int64_t ld, const void* cos_f32, const void* sin_f32,
                                        int64_t batch, int64_t t, int64_t heads, int64_t kv_heads, int64_t head_dim,
                                        void* q_out_bf16, void* k_cache, void* v_cache, int64_t t_max,
                                        const int64_t* pos_dev, int64_t pos, int32_t* dev_status, void* stream) {
  return plq::launch_rope(true, qkv_bf16, ld, cos_f32, sin_f32, batch, t, heads, kv_heads, head_dim, q_out_bf16, k_cache, v_cache,
                          t_max, pos_dev, pos, dev_status, stream);
}

extern "C" int plq_rope_kv_append_nvfp4_values(const void* qkv_bf16, int64_t ld, const void* cos_f32, const void* sin_f32,
                                               int64_t batch, int64_t t, int64_t heads, int64_t kv_heads, int64_t head_dim,
                                               void* q_out_f32, void* k_cache, void* v_cache, int64_t t_max,
                                               const int64_t* pos_dev, int64_t pos, int64_t ctx, void* k_values_bf16,
                                               void* v_values_bf16, int32_t* dev_status, void* stream) {
  using namespace plq;
  if (ctx < t || ctx > t_max || (pos_dev == nullptr && pos + t > ctx)) return PLQ_ERR_SHAPE;
  if (!k_values_bf16 || !v_values_bf16) return PLQ_ERR_NULL;
  if (!aligned16(k_values_bf16) || !aligned16(v_values_bf16)) return PLQ_ERR_ALIGN;
  if (batch * ctx > (1ll << 31)) return PLQ_ERR_LIMIT;
  return launch_rope(true, qkv_bf16, ld, cos_f32, sin_f32, batch, t, heads, kv_heads, head_dim, q_out_f32, k_cache, v_cache, t_max,
                     pos_dev, pos, dev_status, stream, ctx, k_values_bf16, v_values_bf16);
}

extern "C" int plq_unpack_head_rows(const void* k_rows, const void* v_rows, int64_t batch, int64_t t, int64_t t_max,
                                    int64_t kv_heads, void* k_bf16, void* v_bf16, void* stream) {
  using namespace plq;
  if (batch < 0 || t < 0 || kv_heads < 1 || t > t_max) return PLQ_ERR_SHAPE;
  if (batch * t > (1ll << 31) || kv_heads > 4096) return PLQ_ERR_LIMIT;
  if (batch == 0 || t == 0) return PLQ_OK;
  if (!k_rows || !v_rows || !k_bf16 || !v_bf16) return PLQ_ERR_NULL;
  if (!aligned16(k_rows) || !aligned16(v_rows) || !aligned16(k_bf16) || !aligned16(v_bf16)) return PLQ_ERR_ALIGN;
  int st = device_check();
  if (st != PLQ_OK) return st;
  const UnpackRowsArgs a = unpack_args(k_rows, v_rows, batch, t, t_max, kv_heads, k_bf16, v_bf16);
  const long long blocks = (2 * a.total + 255) / 256;
  if (blocks > 0x7FFFFFFF) return PLQ_ERR_LIMIT;
  return launch_overlapped(unpack_head_rows_kernel, dim3(static_cast<unsigned>(blocks)), a, stream);
}
