// Operand pre-passes of the fp32 layers on the tensor cores.
//
// The tcgen05 GEMMs multiply bf16 operands and accumulate in fp32.  An fp32 operand v is fed as
// kPlanes bf16 "planes" p0 = RN_bf16(v), p1 = RN_bf16(v - p0), ... (8 significant bits each), and a
// product of two fp32 operands becomes the plane products a0 b0 + a0 b1 + a1 b0.  The DAC codes of
// the inputs are small integers and exact in a single bf16 plane, so the forward GEMM and the
// weight gradient need only the planes of their other operand.
#include "analog_math.cuh"
#include "device_fast.cuh"
#include "internal.h"

namespace al {

namespace {

__device__ __forceinline__ void split_planes(float v, uint16_t b[kPlanes]) {
#pragma unroll
  for (int p = 0; p < kPlanes; ++p) {
    b[p] = f32_to_bf16_bits(v);
    v = fsub(v, bf16_bits_to_f32(b[p]));  // exact: the difference fits the remaining significant bits
  }
}

// four floats from index 4 v on; `aligned`: the array starts on a 16-byte boundary
__device__ __forceinline__ float4 load_four(const float* __restrict__ src, int64_t v, bool aligned) {
  if (aligned) return reinterpret_cast<const float4*>(src)[v];
  return make_float4(src[v * 4], src[v * 4 + 1], src[v * 4 + 2], src[v * 4 + 3]);
}

// planes[p][e] of src[e], e < count (count is a multiple of 4 on this path: K % 8 == 0)
__global__ void __launch_bounds__(256)
split_planes_kernel(const float* __restrict__ src, int64_t count4, uint16_t* __restrict__ planes, int64_t plane_stride,
                    bool aligned) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < count4; v += (int64_t)gridDim.x * blockDim.x) {
    const float4 x = load_four(src, v, aligned);
    const float in[4] = {x.x, x.y, x.z, x.w};
    uint16_t b[kPlanes][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint16_t bp[kPlanes];
      split_planes(in[i], bp);
#pragma unroll
      for (int p = 0; p < kPlanes; ++p) b[p][i] = bp[p];
    }
#pragma unroll
    for (int p = 0; p < kPlanes; ++p)
      *reinterpret_cast<uint2*>(planes + p * plane_stride + v * 4) =
          make_uint2((uint32_t)b[p][0] | ((uint32_t)b[p][1] << 16), (uint32_t)b[p][2] | ((uint32_t)b[p][3] << 16));
  }
}

// Planes of the upstream gradient, one set per analog tile: planes[(t * kPlanes + p)][m][n] of
//   g[m, n] * keep_t(m, n) * scale(m, t)
// keep_t: the ADC clamp mask of tile t (null: all kept); scale: the DAC step of (row m, tile t)
// (ir null: 1), computed from the saved input range with the function the DAC itself used, so that
// scale * code is the de-quantised input the reference multiplies with.  One thread per 4 columns
// (N % 8 == 0), tiles in gridDim.y.
__global__ void __launch_bounds__(256)
split_planes_grad_kernel(const float* __restrict__ g, int M, int N, const uint32_t* __restrict__ keep_mask, int mask_words,
                   const float* __restrict__ ir, int ir_per_row, float inp_res, uint16_t* __restrict__ planes, bool aligned) {
  const int t = blockIdx.y;
  const int64_t quads = (int64_t)M * (N / 4);
  const int64_t plane_stride = (int64_t)M * N;
  uint16_t* out = planes + (int64_t)t * kPlanes * plane_stride;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < quads; v += (int64_t)gridDim.x * blockDim.x) {
    const int m = (int)(v / (N / 4)), n = (int)(v % (N / 4)) * 4;
    const float4 x = load_four(g, v, aligned);
    float in[4] = {x.x, x.y, x.z, x.w};
    float scale = 1.0f;
    if (ir != nullptr) scale = quant_step<kF32>(ir[ir_per_row ? (int64_t)t * M + m : t], inp_res);
    uint32_t word = 0xffffffffu;
    if (keep_mask != nullptr) word = keep_mask[((int64_t)t * mask_words + (n >> 5)) * M + m];
    uint16_t b[kPlanes][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float val = ((word >> ((n & 31) + i)) & 1u) ? in[i] : 0.0f;
      if (ir != nullptr) val = fmul(val, scale);
      uint16_t bp[kPlanes];
      split_planes(val, bp);
#pragma unroll
      for (int p = 0; p < kPlanes; ++p) b[p][i] = bp[p];
    }
#pragma unroll
    for (int p = 0; p < kPlanes; ++p)
      *reinterpret_cast<uint2*>(out + p * plane_stride + v * 4) =
          make_uint2((uint32_t)b[p][0] | ((uint32_t)b[p][1] << 16), (uint32_t)b[p][2] | ((uint32_t)b[p][3] << 16));
  }
}

// ---- DAC and weight pass of these layers -----------------------------------------------------------------------
// Both write what the GEMMs read and nothing else: the codes (2 bytes an element; the general pass also wrote the
// quantised inputs, 4 more) and the planes of the modified weights (the general pass wrote them as fp32 for
// split_planes_kernel to read back).  One warp per (row, tile) segment, eight consecutive elements per lane and step --
// one call of the noise generator -- held in registers between the abs-max and their use.  4096 x 4096: DAC 29 -> 21 us,
// weights with noise 38 + 20 -> 32 us.  Tiles and K are multiples of 8 and bases 16-byte aligned (checked by the host).
constexpr int kSegWarps = 8;
constexpr int kHeld = 4;  // groups of eight a lane keeps: tiles of up to 1024 (wider ones are read a second time)

struct Eight {
  float v[8];
};
__device__ __forceinline__ Eight load_eight(const float* p, bool on) {
  Eight r;
  const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float4 a = on ? __ldg(reinterpret_cast<const float4*>(p)) : z, b = on ? __ldg(reinterpret_cast<const float4*>(p) + 1) : z;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}
__device__ __forceinline__ float abs_max_eight(const Eight& e, float m) {
#pragma unroll
  for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(e.v[i]));
  return m;
}
__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}
__device__ __forceinline__ uint4 pack_eight(const uint16_t b[8]) {
  return make_uint4((uint32_t)b[0] | ((uint32_t)b[1] << 16), (uint32_t)b[2] | ((uint32_t)b[3] << 16),
                    (uint32_t)b[4] | ((uint32_t)b[5] << 16), (uint32_t)b[6] | ((uint32_t)b[7] << 16));
}

__global__ void __launch_bounds__(kSegWarps * 32)
dac_codes_kernel(const float* __restrict__ x, int M, int K, int T, int tile_w, int ir_mode, const float* __restrict__ ir_static,
                 float inp_res, uint16_t* __restrict__ codes, float* __restrict__ ir_rows, uint32_t* __restrict__ zero_words,
                 int zero_count) {
  if (blockIdx.x == 0 && (int)threadIdx.x < zero_count) zero_words[threadIdx.x] = 0u;  // for the weight pass behind
  const unsigned seg = blockIdx.x * kSegWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (seg >= (unsigned)M * (unsigned)T) return;
  const int m = (int)(seg / (unsigned)T), t = (int)(seg - (unsigned)m * (unsigned)T), groups = tile_w / 8;
  const float* const src = x + (int64_t)m * K + (int64_t)t * tile_w;
  uint16_t* const dst = codes + (int64_t)m * K + (int64_t)t * tile_w;
  Eight held[kHeld];
#pragma unroll
  for (int j = 0; j < kHeld; ++j) held[j] = load_eight(src + (j * 32 + lane) * 8, j * 32 + lane < groups);
  float ir;
  if (ir_mode == AL_IR_DYNAMIC) {
    float mx = 0.0f;
#pragma unroll
    for (int j = 0; j < kHeld; ++j) mx = abs_max_eight(held[j], mx);
    for (int g = kHeld * 32 + lane; g < groups; g += 32) mx = abs_max_eight(load_eight(src + g * 8, true), mx);
    ir = warp_max(mx);
    if (lane == 0) ir_rows[(int64_t)t * M + m] = ir;
  } else {
    ir = ir_static[t];
  }
  const QuantSeg q = dac_prepare<kF32>(ir, inp_res, ir_mode != AL_IR_DYNAMIC, false);
  const auto put = [&](int g, const Eight& e) {
    uint16_t b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float code;
      dac_apply<kF32>(q, e.v[i], &code);
      b[i] = f32_to_bf16_bits(code);  // a small integer: exact
    }
    *reinterpret_cast<uint4*>(dst + g * 8) = pack_eight(b);
  };
#pragma unroll
  for (int j = 0; j < kHeld; ++j)
    if (j * 32 + lane < groups) put(j * 32 + lane, held[j]);
  for (int g = kHeld * 32 + lane; g < groups; g += 32) put(g, load_eight(src + g * 8, true));
}

// planes of w + (std_dev * segment abs-max) * xi; w_mod (nullable) receives the fp32 sum as well
__global__ void __launch_bounds__(kSegWarps * 32)
weight_planes_kernel(const float* __restrict__ w, int N, int K, int T, int tile_w, float* __restrict__ w_amax,
                     float* __restrict__ tile_max, int noise_type, float std_dev, const NoiseKeys nk,
                     uint16_t* __restrict__ planes, float* __restrict__ w_mod) {
  const unsigned seg = blockIdx.x * kSegWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (seg >= (unsigned)N * (unsigned)T) return;
  const int n = (int)(seg / (unsigned)T), t = (int)(seg - (unsigned)n * (unsigned)T), groups = tile_w / 8;
  const int64_t start = (int64_t)n * K + (int64_t)t * tile_w, plane_stride = (int64_t)N * K;
  Eight held[kHeld];
#pragma unroll
  for (int j = 0; j < kHeld; ++j) held[j] = load_eight(w + start + (j * 32 + lane) * 8, j * 32 + lane < groups);
  float mx = 0.0f;
#pragma unroll
  for (int j = 0; j < kHeld; ++j) mx = abs_max_eight(held[j], mx);
  for (int g = kHeld * 32 + lane; g < groups; g += 32) mx = abs_max_eight(load_eight(w + start + g * 8, true), mx);
  mx = warp_max(mx);
  if (lane == 0) {
    w_amax[(int64_t)t * N + n] = mx;
    unsigned int* const slot = reinterpret_cast<unsigned int*>(tile_max) + t;
    const unsigned int bits = __float_as_uint(mx);
    if (bits > *reinterpret_cast<volatile unsigned int*>(slot)) atomicMax(slot, bits);
  }
  const WeightSeg ws = weight_prepare<kF32>(AL_QUANT_NONE, mx, 1.0f, 1.0f, false, noise_type, std_dev, mx, false);
  const NoiseCounter ctr = noise_counter(nk);
  const auto put = [&](int g, Eight e) {
    if (ws.noise) {
      float z[8];
      normal8_keyed(nk, ctr, (uint64_t)(start + g * 8) >> 3, z);
#pragma unroll
      for (int i = 0; i < 8; ++i) e.v[i] = weight_apply<kF32>(ws, e.v[i], z[i]);
    }
    uint16_t b[kPlanes][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint16_t bp[kPlanes];
      split_planes(e.v[i], bp);
#pragma unroll
      for (int p = 0; p < kPlanes; ++p) b[p][i] = bp[p];
    }
#pragma unroll
    for (int p = 0; p < kPlanes; ++p) *reinterpret_cast<uint4*>(planes + p * plane_stride + start + g * 8) = pack_eight(b[p]);
    if (w_mod != nullptr) {
      float4* const out = reinterpret_cast<float4*>(w_mod + start + g * 8);
      out[0] = make_float4(e.v[0], e.v[1], e.v[2], e.v[3]);
      out[1] = make_float4(e.v[4], e.v[5], e.v[6], e.v[7]);
    }
  };
#pragma unroll
  for (int j = 0; j < kHeld; ++j)
    if (j * 32 + lane < groups) put(j * 32 + lane, held[j]);
  for (int g = kHeld * 32 + lane; g < groups; g += 32) put(g, load_eight(w + start + g * 8, true));
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
unsigned grid_for(int64_t work_items) {
  const int64_t blocks = (work_items + 255) / 256;
  return (unsigned)(blocks < 148 * 16 ? (blocks < 1 ? 1 : blocks) : 148 * 16);
}

}  // namespace

int launch_dac_codes(const float* x, int M, int K, const TileTable& tt, int ir_mode, const float* ir_static, float inp_res,
                     void* codes16, float* ir_rows, cudaStream_t s, void* zero_words, int zero_count, bool* zeroed) {
  ProfScope prof(AL_K_DAC, s);
  if (zero_words == nullptr || zero_count > kSegWarps * 32) zero_count = 0;
  *zeroed = zero_count > 0;
  const unsigned blocks = (unsigned)(((int64_t)M * tt.T + kSegWarps - 1) / kSegWarps);
  dac_codes_kernel<<<blocks, kSegWarps * 32, 0, s>>>(x, M, K, tt.T, tt.hi(0), ir_mode, ir_static, inp_res,
                                                     static_cast<uint16_t*>(codes16), ir_rows,
                                                     static_cast<uint32_t*>(zero_words), zero_count);
  return check_launch("dac_codes");
}

int launch_weight_planes(const float* w, int N, int K, const TileTable& tt, float* w_amax, float* tile_max, int noise_type,
                         float std_dev, uint64_t seed, uint64_t offset, const uint64_t* offset_base, void* planes,
                         float* w_mod, cudaStream_t s, bool tile_max_zeroed) {
  ProfScope prof(AL_K_WEIGHT_MODIFY, s);
  const cudaError_t e = tile_max_zeroed ? cudaSuccess : cudaMemsetAsync(tile_max, 0, 2 * sizeof(float) * tt.T, s);
  if (e != cudaSuccess) {
    set_error("weight_planes: memset: %s", cudaGetErrorString(e));
    return AL_ERR_CUDA;
  }
  const unsigned blocks = (unsigned)(((int64_t)N * tt.T + kSegWarps - 1) / kSegWarps);
  weight_planes_kernel<<<blocks, kSegWarps * 32, 0, s>>>(w, N, K, tt.T, tt.hi(0), w_amax, tile_max, noise_type, std_dev,
                                                         make_noise_keys(seed, offset, 0u, offset_base),
                                                         static_cast<uint16_t*>(planes), w_mod);
  return check_launch("weight_planes");
}

int launch_split_planes(const float* src, int64_t count, void* planes, cudaStream_t s) {
  ProfScope prof(AL_K_WEIGHT_MODIFY, s);
  split_planes_kernel<<<grid_for(count / 4), 256, 0, s>>>(src, count / 4, static_cast<uint16_t*>(planes), count,
                                                         aligned16(src));
  return check_launch("split_planes");
}

int launch_split_planes_grad(const float* g, int M, int N, const uint32_t* keep_mask, int mask_words, const float* ir,
                       int ir_per_row, float inp_res, int sets, void* planes, cudaStream_t s) {
  ProfScope prof(AL_K_DAC, s);
  dim3 grid(grid_for((int64_t)M * (N / 4)), sets);
  split_planes_grad_kernel<<<grid, 256, 0, s>>>(g, M, N, keep_mask, mask_words, ir, ir_per_row, inp_res,
                                          static_cast<uint16_t*>(planes), aligned16(g));
  return check_launch("split_planes_grad");
}

}  // namespace al
