// Operands of bf16 layers whose sizes TMA cannot address (a tile width, K or N that is no multiple of 8): the
// pre-passes that read every operand anyway write it in a pitched layout the tcgen05 GEMMs can load.
//
//   [rows, K]  ->  [rows, T * wp]   analog tile t starts at column t * wp, wp = widest tile rounded up to 8
//   [M, N]     ->  [M, np]          np = N rounded up to 8 (the upstream gradient of a backward pass)
//
// Padding columns hold zeros.  The destination is 16-byte aligned at every tile start; the source is not, so a
// lane builds its 16-byte vector from two aligned loads and a funnel shift (all chunks of a segment share the
// shift).  The second load hits L1: the passes stay bound by one trip through memory.
// Values are those of the dense pre-passes (prepass_kernels.cu), noise included: the generator is addressed by the
// element's index in the dense matrix.
// 1000 x 2500 inputs: 5.6 us, as the dense pass; 1500 x 2500 weights with noise: 15.6 us against 11.4 us of the dense
// pass (the generator runs for the straddled groups of lane 31 a second time).
#include "analog_math.cuh"
#include "device_fast.cuh"
#include "internal.h"

namespace al {

namespace {

constexpr int kWarps = 8;

// A bf16 array that is read in 16-byte vectors at any element offset.
struct Source {
  const uint16_t* base;  // aligned down to 16 bytes
  int lead;              // elements between base and the array's first
  int64_t end;           // lead + number of elements: vectors that end beyond are read by element
};
__device__ __forceinline__ Source make_source(const uint16_t* p, int64_t count) {
  Source s;
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  s.lead = (int)((a & 15) >> 1);
  s.base = reinterpret_cast<const uint16_t*>(a & ~(uintptr_t)15);
  s.end = s.lead + count;
  return s;
}

// 8 elements from two neighbouring vectors, `r` elements into the first
__device__ __forceinline__ uint4 funnel8(const uint4& a, const uint4& b, int r) {
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (r & 4) {
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
  }
  if (r & 2) {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
  }
  if (r & 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// keeps the first n elements of a vector (n may be <= 0 or >= 8), the others become zero
__device__ __forceinline__ uint4 first_n(uint4 v, int n) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = 2 * i + 1 < n ? w[i] : (2 * i < n ? w[i] & 0xffffu : 0u);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// elements [e, e + 8) of the array, those from e + n on as zero
__device__ __forceinline__ uint4 load8(const Source& s, int64_t e, int n) {
  const int64_t a = e + s.lead;
  const int r = (int)(a & 7);
  const int64_t v = a - r;
  if (n <= 0) return make_uint4(0u, 0u, 0u, 0u);
  if (v >= s.lead && v + (r ? 16 : 8) <= s.end) {
    const uint4 lo = __ldg(reinterpret_cast<const uint4*>(s.base + v));
    const uint4 hi = r ? __ldg(reinterpret_cast<const uint4*>(s.base + v + 8)) : lo;
    return first_n(funnel8(lo, hi, r), n);
  }
  uint32_t w[4] = {0u, 0u, 0u, 0u};  // the first and the last vectors of the array
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i < n) w[i >> 1] |= (uint32_t)__ldg(s.base + a + i) << (16 * (i & 1));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ float vec_abs_max(const uint4& v, float m) {
  __nv_bfloat162 m2 = __hmax2(__habs2(as_bf162(v.x)), __habs2(as_bf162(v.y)));
  m2 = __hmax2(m2, __hmax2(__habs2(as_bf162(v.z)), __habs2(as_bf162(v.w))));
  return fmaxf(m, fmaxf(__low2float(m2), __high2float(m2)));
}
__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

__device__ __forceinline__ uint4 dac_vec(const uint4& raw, const QuantSeg& q, bool packed) {
  uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  if (packed) {  // the bf16x2 form of dac_kernel
    const __nv_bfloat162 b2 = __float2bfloat162_rn(q.bound), nb2 = __float2bfloat162_rn(-q.bound);
    const __nv_bfloat162 step2 = __float2bfloat162_rn(q.step);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 x2 = as_bf162(w[i]);
      if (q.clampit) x2 = __hmin2_nan(__hmax2_nan(x2, nb2), b2);
      const __nv_bfloat162 q2 = __floats2bfloat162_rn(fdiv_rcp(__low2float(x2), q.stepc, q.rstep),
                                                      fdiv_rcp(__high2float(x2), q.stepc, q.rstep));
      const float lo = rint_small(__low2float(q2)), hi = rint_small(__high2float(q2));
      w[i] = as_u32(__hmul2_rn(as_bf162(__byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632)), step2));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float code;
      const uint32_t lo = f32_to_bf16_bits(dac_apply<kBF16>(q, __uint_as_float(w[i] << 16), &code));
      const uint32_t hi = f32_to_bf16_bits(dac_apply<kBF16>(q, __uint_as_float(w[i] & 0xffff0000u), &code));
      w[i] = lo | (hi << 16);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

constexpr int kHeld = 4;  // vectors a lane keeps between the range and the quantisation: tiles of up to 1024

// xq[m, t * wp + i] = DAC(x[m, lo_t + i]), one warp per (row, tile)
__global__ void __launch_bounds__(kWarps * 32)
dac_ragged_kernel(const uint16_t* __restrict__ x, int M, int K, RaggedTiles rt, int ir_mode,
                  const uint16_t* __restrict__ ir_static, float inp_res, int no_rounding, int small_codes,
                  uint16_t* __restrict__ xq, uint16_t* __restrict__ ir_rows) {
  const unsigned seg = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (seg >= (unsigned)M * (unsigned)rt.T) return;
  const int m = (int)(seg / (unsigned)rt.T), t = (int)(seg - (unsigned)m * (unsigned)rt.T);
  const int len = rt.width(t), chunks = rt.pitch / 8;
  const Source src = make_source(x, (int64_t)M * K);
  const int64_t start = (int64_t)m * K + rt.lo(t);
  uint4 held[kHeld];
  float mx = 0.0f;
#pragma unroll
  for (int j = 0; j < kHeld; ++j) {
    const int c = j * 32 + lane;
    held[j] = load8(src, start + c * 8, len - c * 8);
  }
  float ir = 0.0f;
  bool clampit = false;
  if (ir_mode == AL_IR_DYNAMIC) {
#pragma unroll
    for (int j = 0; j < kHeld; ++j) mx = vec_abs_max(held[j], mx);
    for (int c = kHeld * 32 + lane; c < chunks; c += 32) mx = vec_abs_max(load8(src, start + c * 8, len - c * 8), mx);
    ir = warp_max(mx);
    if (lane == 0) ir_rows[(int64_t)t * M + m] = f32_to_bf16_bits(ir);
  } else if (ir_mode == AL_IR_STATIC) {
    ir = bf16_bits_to_f32(ir_static[t]);
    clampit = true;
  }
  const QuantSeg q = dac_prepare<kBF16>(ir, inp_res, clampit, no_rounding != 0);
  const bool packed = q.quantise && !q.no_rounding && small_codes;
  uint16_t* dst = xq + (int64_t)m * rt.T * rt.pitch + (int64_t)t * rt.pitch;
#pragma unroll
  for (int j = 0; j < kHeld; ++j) {
    const int c = j * 32 + lane;
    if (c < chunks) *reinterpret_cast<uint4*>(dst + c * 8) = first_n(dac_vec(held[j], q, packed), len - c * 8);
  }
  for (int c = kHeld * 32 + lane; c < chunks; c += 32)
    *reinterpret_cast<uint4*>(dst + c * 8) =
        first_n(dac_vec(load8(src, start + c * 8, len - c * 8), q, packed), len - c * 8);
}

// Weight pre-pass: out[n, t * wp + i] = noise(discretise(w[n, lo_t + i])), one warp per (channel, tile).
// FUSED (the pass of launch_weight_fused): abs-max and tile maximum are taken here, the only modifier is noise on
// the scale of the segment's own abs-max.  Otherwise (launch_weight_modify) both arrive in w_amax / tile_max.
struct WeightRagged {
  const uint16_t* w;
  int N, K;
  RaggedTiles rt;
  uint16_t* w_amax;
  float* tile_max;
  const int32_t* flags;
  int quant_type, noise_type, no_rounding, aligned;
  float n_states, max_state, std_dev;
  uint64_t seed, offset;
  const uint64_t* offset_base;
  uint16_t* out;
};

// the normals of elements [8 group, 8 group + 8) as the dense pass draws them, rounded to bf16
template <bool FUSED>
__device__ __forceinline__ uint4 group_noise(uint64_t seed, uint64_t offset, int64_t group, int64_t start, int64_t end,
                                             bool aligned) {
  float z[8];
  if (FUSED && aligned && group * 8 >= start && group * 8 + 8 <= end) {
    normal8_fast(seed, offset, 0u, (uint64_t)group, z);  // whole groups of a segment
  } else {                                               // its ragged ends (and the separate modifier pass)
    normal4(seed, offset, 0u, (uint64_t)group * 2, z);
    normal4(seed, offset, 0u, (uint64_t)group * 2 + 1, z + 4);
  }
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = as_u32(__floats2bfloat162_rn(z[2 * i], z[2 * i + 1]));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <bool FUSED>
__global__ void __launch_bounds__(kWarps * 32) weight_ragged_kernel(const WeightRagged p) {
  const unsigned seg = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (seg >= (unsigned)p.N * (unsigned)p.rt.T) return;
  const int n = (int)(seg / (unsigned)p.rt.T), t = (int)(seg - (unsigned)n * (unsigned)p.rt.T);
  const int len = p.rt.width(t), chunks = p.rt.pitch / 8;
  const Source src = make_source(p.w, (int64_t)p.N * p.K);
  const int64_t start = (int64_t)n * p.K + p.rt.lo(t);
  const uint64_t offset = p.offset + (p.offset_base != nullptr ? *p.offset_base : 0ull);
  uint4 held[kHeld];
#pragma unroll
  for (int j = 0; j < kHeld; ++j) {
    const int c = j * 32 + lane;
    held[j] = load8(src, start + c * 8, len - c * 8);
  }
  WeightSeg ws;
  if (FUSED) {
    float mx = 0.0f;
#pragma unroll
    for (int j = 0; j < kHeld; ++j) mx = vec_abs_max(held[j], mx);
    for (int c = kHeld * 32 + lane; c < chunks; c += 32) mx = vec_abs_max(load8(src, start + c * 8, len - c * 8), mx);
    mx = warp_max(mx);
    if (lane == 0 && p.tile_max != nullptr) {
      p.w_amax[(int64_t)t * p.N + n] = f32_to_bf16_bits(mx);
      unsigned int* slot = reinterpret_cast<unsigned int*>(p.tile_max) + t;
      const unsigned int bits = __float_as_uint(mx);
      if (bits > *reinterpret_cast<volatile unsigned int*>(slot)) atomicMax(slot, bits);
    }
    ws = weight_prepare<kBF16>(AL_QUANT_NONE, mx, 1.0f, 1.0f, false, p.noise_type, p.std_dev, mx, false);
  } else {
    const float row_max = bf16_bits_to_f32(p.w_amax[(int64_t)t * p.N + n]);
    const float t_max = rnd<kBF16>(p.tile_max[t]);
    const float n_scale = p.noise_type == AL_NOISE_ADD_NORMAL ? t_max : row_max;
    ws = p.quant_type == kQuantLearnClamp
             ? weight_prepare_learn_clamp<kBF16>(row_max, p.flags[t] != 0, p.noise_type, p.std_dev, n_scale)
             : weight_prepare<kBF16>(p.quant_type, p.quant_type == AL_QUANT_DISCRETIZE ? t_max : row_max, p.n_states,
                                     p.max_state, p.flags[t] != 0, p.noise_type, p.std_dev, n_scale, p.no_rounding != 0);
  }
  const int r = (int)(start & 7);
  const int64_t g0 = start >> 3, seg_end = start + len;
  uint16_t* dst = p.out + (int64_t)n * p.rt.T * p.rt.pitch + (int64_t)t * p.rt.pitch;
  auto modify = [&](int c, uint4 raw) {  // called by whole warps
    uint4 z = make_uint4(0u, 0u, 0u, 0u);
    if (ws.noise) {
      // a chunk straddles two groups of the noise stream unless the segment starts on one: the second is the
      // next lane's first
      z = group_noise<FUSED>(p.seed, offset, g0 + c, start, seg_end, p.aligned != 0);
      uint4 nx;
      nx.x = __shfl_down_sync(0xffffffffu, z.x, 1);
      nx.y = __shfl_down_sync(0xffffffffu, z.y, 1);
      nx.z = __shfl_down_sync(0xffffffffu, z.z, 1);
      nx.w = __shfl_down_sync(0xffffffffu, z.w, 1);
      if (r != 0) {
        if (lane == 31 && c < chunks) nx = group_noise<FUSED>(p.seed, offset, g0 + c + 1, start, seg_end, p.aligned != 0);
        z = funnel8(z, nx, r);
      }
    }
    if (c >= chunks) return;
    uint32_t wv[4] = {raw.x, raw.y, raw.z, raw.w}, zv[4] = {z.x, z.y, z.z, z.w};
    if (ws.quant) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t lo = f32_to_bf16_bits(weight_apply<kBF16>(ws, __uint_as_float(wv[i] << 16), __uint_as_float(zv[i] << 16)));
        const uint32_t hi = f32_to_bf16_bits(
            weight_apply<kBF16>(ws, __uint_as_float(wv[i] & 0xffff0000u), __uint_as_float(zv[i] & 0xffff0000u)));
        wv[i] = lo | (hi << 16);
      }
    } else if (ws.noise) {
      const __nv_bfloat162 amp2 = __float2bfloat162_rn(ws.amp);
#pragma unroll
      for (int i = 0; i < 4; ++i) wv[i] = as_u32(__hadd2_rn(as_bf162(wv[i]), __hmul2_rn(amp2, as_bf162(zv[i]))));
    }
    *reinterpret_cast<uint4*>(dst + c * 8) = first_n(make_uint4(wv[0], wv[1], wv[2], wv[3]), len - c * 8);
  };
#pragma unroll
  for (int j = 0; j < kHeld; ++j)
    if (j * 32 < chunks) modify(j * 32 + lane, held[j]);
  for (int c0 = kHeld * 32; c0 < chunks; c0 += 32)
    modify(c0 + lane, load8(src, start + (c0 + lane) * 8, len - (c0 + lane) * 8));
}

// dst[m, 0 .. np) = src[m, 0 .. N), zeros behind; one thread per 16-byte vector
__global__ void __launch_bounds__(256)
pitch_rows_kernel(const uint16_t* __restrict__ src, int64_t M, int N, int vecs, uint16_t* __restrict__ dst) {
  const Source s = make_source(src, M * N);
  const int64_t total = M * vecs;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < total; v += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = v / vecs;
    const int c = (int)(v - m * vecs);
    reinterpret_cast<uint4*>(dst)[v] = load8(s, m * N + c * 8, N - c * 8);
  }
}

inline unsigned seg_blocks(int64_t segs) { return (unsigned)((segs + kWarps - 1) / kWarps); }

}  // namespace

bool ragged_tiles(const TileTable& tt, RaggedTiles* out) {
  const int last = tt.hi(tt.T - 1) - tt.lo(tt.T - 1), first = tt.hi(0);
  out->T = tt.T;
  out->base = last;
  out->extra = first == last ? 0 : tt.hi(tt.T - 1) - tt.T * last;
  out->pitch = (first + 7) / 8 * 8;
  for (int t = 0; t < tt.T; ++t)
    if (out->lo(t) != tt.lo(t) || out->width(t) != tt.hi(t) - tt.lo(t)) return false;
  return true;
}

int launch_dac_ragged(const void* x, int M, int K, const RaggedTiles& rt, int ir_mode, const void* ir_static,
                      float inp_res, int no_rounding, void* xq, void* ir_rows, cudaStream_t s) {
  ProfScope prof(AL_K_DAC, s);
  const float states = inp_res > 0.0f ? (inp_res > 1.0f ? inp_res : 1.0f / inp_res) : 0.0f;
  dac_ragged_kernel<<<seg_blocks((int64_t)M * rt.T), kWarps * 32, 0, s>>>(
      static_cast<const uint16_t*>(x), M, K, rt, ir_mode, static_cast<const uint16_t*>(ir_static), inp_res, no_rounding,
      states < 4.0e6f, static_cast<uint16_t*>(xq), static_cast<uint16_t*>(ir_rows));
  return check_launch("dac_ragged");
}

int launch_weight_ragged(bool fused, const void* w, int N, int K, const RaggedTiles& rt, void* w_amax, float* tile_max,
                         const int32_t* flags, int quant_type, float n_states, float max_state, int noise_type,
                         float std_dev, uint64_t seed, uint64_t offset, int no_rounding, void* out, cudaStream_t s,
                         const uint64_t* offset_base) {
  ProfScope prof(AL_K_WEIGHT_MODIFY, s);
  if (fused && tile_max != nullptr) {
    cudaError_t e = cudaMemsetAsync(tile_max, 0, 2 * sizeof(float) * rt.T, s);
    if (e != cudaSuccess) {
      set_error("weight_ragged: memset: %s", cudaGetErrorString(e));
      return AL_ERR_CUDA;
    }
  }
  WeightRagged p;
  p.w = static_cast<const uint16_t*>(w);
  p.N = N; p.K = K;
  p.rt = rt;
  p.w_amax = static_cast<uint16_t*>(w_amax);
  p.tile_max = tile_max;
  p.flags = flags;
  p.quant_type = quant_type; p.noise_type = noise_type; p.no_rounding = no_rounding;
  p.aligned = reinterpret_cast<uintptr_t>(w) % 16 == 0;
  p.n_states = n_states; p.max_state = max_state; p.std_dev = std_dev;
  p.seed = seed; p.offset = offset;
  p.offset_base = offset_base;
  p.out = static_cast<uint16_t*>(out);
  const unsigned blocks = seg_blocks((int64_t)N * rt.T);
  if (fused) weight_ragged_kernel<true><<<blocks, kWarps * 32, 0, s>>>(p);
  else weight_ragged_kernel<false><<<blocks, kWarps * 32, 0, s>>>(p);
  return check_launch("weight_ragged");
}

int launch_pitch_rows(const void* src, int M, int N, void* dst, cudaStream_t s) {
  ProfScope prof(AL_K_DAC, s);
  const int vecs = (N + 7) / 8;
  const int64_t blocks = ((int64_t)M * vecs + 255) / 256;
  pitch_rows_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s>>>(
      static_cast<const uint16_t*>(src), M, N, vecs, static_cast<uint16_t*>(dst));
  return check_launch("pitch_rows");
}

}  // namespace al
