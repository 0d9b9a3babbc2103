// Element-wise and reduction parts of the backward pass: the bias gradient (column sums of
// the upstream gradient) and, for learned/fixed input ranges, the input-range gradient with
// its decay term followed by the straight-through zeroing of clipped inputs.  Both reduce in
// a fixed order (no floating-point atomics).
#include <cooperative_groups.h>

#include "analog_math.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace al {

namespace {

// Column sums of g [M, N].  A cluster of kBiasCluster CTAs owns COLS columns of every `splits`-th run of rows; a thread
// adds VN columns of its rows in runs of bias_ahead with their loads in flight, then the row groups are added in shared
// memory and the CTAs of the cluster through distributed shared memory, always in the same order.
// Reading g bounds it where the CTAs fill the chip (large N, or a split); otherwise what a few CTAs have in flight.
// A run is summed by itself first: that keeps the chain of roundings shorter than one per 256 rows of the matrix.
constexpr int kBiasCluster = 8, kBiasThreads = 256, kBiasMaxSplits = 32;
// rows of a thread whose loads are in flight
constexpr int bias_ahead(int vn, bool wide) { return wide && vn == 1 ? 16 : 8; }
// Split from this many rows per thread on, and a quarter more for each column group: a second kernel costs about 1.5 us,
// and groups bring CTAs of their own.  Unsplit -> split, fp32: 64 columns 4096 rows (32 per thread) 3.9 -> 4.1 us,
// 8192 5.6 -> 5.1, 131072 57 -> 8.2; 65 columns 131072 100 -> 13; 1001 columns 4096 rows (128) 5.7 -> 6.4; 1000 columns
// 65536 rows (512) 90 -> 43.
constexpr int kBiasSplitRows = 64;
// WIDE: the loads of a last short run are in flight together as well, which takes 51 registers instead of 40 -- for
// grids that leave the SMs room for it.  333 x 777 fp32 3.0 -> 2.5 us, 8192 x 256 6.2 -> 5.2, but 64 x 16384 6.3 -> 10.0
constexpr unsigned kBiasWideGroups = 4 * 148 / kBiasCluster;
constexpr int kBiasCtas = 4 * 148;  // what a split fills the chip with: four of up to eight resident CTAs per SM
template <int DT, int VN>
__device__ __forceinline__ void load_cols(const void* p, int64_t idx, float v[VN]) {
  if (VN == 1) {
    v[0] = Elem<DT>::load(p, idx);
  } else if (DT == kF32) {
    const float4 f = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + idx);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p) + idx);
    v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
    v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
  }
}
template <int DT, int VN, int COLS, bool WIDE, bool SPLIT>
__global__ void __cluster_dims__(1, kBiasCluster, 1) __launch_bounds__(kBiasThreads)
bias_grad_kernel(const void* __restrict__ g, int M, int N, int splits, float* __restrict__ partial,
                 void* __restrict__ grad_bias) {
  constexpr int kColThreads = COLS / VN, kRowThreads = kBiasThreads / kColThreads, kAhead = bias_ahead(VN, WIDE);
  __shared__ float part[kRowThreads][COLS];
  __shared__ float total[COLS];
  const int tc = threadIdx.x % kColThreads, tr = threadIdx.x / kColThreads;
  const int n = blockIdx.x * COLS + tc * VN;  // N % VN == 0
  float s[VN];
#pragma unroll
  for (int i = 0; i < VN; ++i) s[i] = 0.0f;
  const int step = kRowThreads * kBiasCluster * (SPLIT ? splits : 1), first = (int)blockIdx.y * kRowThreads + tr;
  if (n < N && first < M) {
    const int count = (M - 1 - first) / step + 1;  // rows of this thread; no row index below goes beyond M
    int r = 0;
    for (; WIDE ? r < count : r + kAhead <= count; r += kAhead) {
      float v[kAhead][VN];
      if (!WIDE || r + kAhead <= count) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) load_cols<DT, VN>(g, (int64_t)(first + (r + u) * step) * N + n, v[u]);
      } else {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (r + u < count) {
            load_cols<DT, VN>(g, (int64_t)(first + (r + u) * step) * N + n, v[u]);
          } else {
#pragma unroll
            for (int i = 0; i < VN; ++i) v[u][i] = 0.0f;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < VN; ++i) {
        float run = v[0][i];
#pragma unroll
        for (int u = 1; u < kAhead; ++u) run = fadd(run, v[u][i]);
        s[i] = fadd(s[i], run);
      }
    }
    for (; !WIDE && r < count; ++r) {
      float v[VN];
      load_cols<DT, VN>(g, (int64_t)(first + r * step) * N + n, v);
#pragma unroll
      for (int i = 0; i < VN; ++i) s[i] = fadd(s[i], v[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < VN; ++i) part[tr][tc * VN + i] = s[i];
  __syncthreads();
  if (threadIdx.x < COLS) {
    float sum = part[0][threadIdx.x];
#pragma unroll
    for (int r = 1; r < kRowThreads; ++r) sum = fadd(sum, part[r][threadIdx.x]);
    total[threadIdx.x] = sum;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int col = blockIdx.x * COLS + threadIdx.x;
  if (blockIdx.y % kBiasCluster == 0 && threadIdx.x < COLS && col < N) {
    float sum = total[threadIdx.x];
#pragma unroll
    for (int c = 1; c < kBiasCluster; ++c) sum = fadd(sum, cluster.map_shared_rank(total, c)[threadIdx.x]);
    if (!SPLIT) Elem<DT>::store(grad_bias, col, sum);
    else partial[(int64_t)(blockIdx.y / kBiasCluster) * N + col] = sum;
  }
  cluster.sync();  // no CTA leaves while another still reads its sums
}
template <int DT>
__global__ void __launch_bounds__(kBiasThreads)
bias_sum_kernel(const float* __restrict__ partial, int splits, int N, void* __restrict__ grad_bias) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float sum = partial[n];
  for (int c = 1; c < splits; ++c) sum = fadd(sum, partial[(int64_t)c * N + n]);
  Elem<DT>::store(grad_bias, n, sum);
}

// Partial sums for the range gradient, then zero grad_x where the input was clipped and does not sit exactly on
// the range.  A block takes `block_rows` consecutive rows of one tile and writes three partial sums: fp32 within a lane's
// share of one row, double beyond it (terms of both signs cancel in fast mode), kept as the sum of two floats because
// the workspace is only known to be aligned for those.  Bound by reading x and grad_x once.  VEC: every (row, tile) segment starts and ends on a 16-byte boundary (the launcher
// checked), so a lane moves 16-byte vectors; single elements otherwise.
struct IrSums {
  float up, lo, cnt;
};
// one element: sums, and whether its gradient is blocked
__device__ __forceinline__ bool ir_element(float xv, float gv, float ir, int fast_mode, IrSums& s) {
  if (fast_mode) {
    // plain clamp with tensor bounds: the bounds collect the gradient outside [-ir, ir]
    const bool up = xv > ir, dn = xv < -ir;
    if (up) s.up += gv;
    if (dn) s.lo += gv;
    return up || dn;
  }
  const bool up = xv >= ir, dn = xv <= -ir;
  if (up) s.up += fminf(gv, 0.0f);
  if (dn) s.lo += fmaxf(gv, 0.0f);
  if (!(up || dn)) return false;
  s.cnt += 1.0f;
  return fabsf(xv) != ir;
}
template <int DT, bool VEC>
__global__ void __launch_bounds__(256)
static_ir_partial_kernel(const void* __restrict__ x, const void* __restrict__ ir_used,
                         void* __restrict__ grad_x, int M, int K, TileTable tt,
                         float* __restrict__ partial, int fast_mode, int block_rows) {
  __shared__ double part[8][3];
  const int t = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lo = tt.lo(t), len = tt.hi(t) - lo;
  const float ir = Elem<DT>::load(ir_used, t);
  double up = 0.0, down = 0.0;
  IrSums s = {0.0f, 0.0f, 0.0f};  // up, lo: of the row at hand; cnt: of all rows (exact)
  const unsigned m_first = blockIdx.x * (unsigned)block_rows, m_end = min((unsigned)M, m_first + (unsigned)block_rows);
  for (unsigned m = m_first + warp; m < m_end; m += 8) {
    s.up = s.lo = 0.0f;
    const int64_t start = (int64_t)m * K + lo;
    if (VEC) {
      constexpr int VN = DT == kF32 ? 4 : 8;
      constexpr int ES = 16 / VN;
      const uint4* xv = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(x) + start * ES);
      uint4* gv = reinterpret_cast<uint4*>(reinterpret_cast<char*>(grad_x) + start * ES);
      const int nvec = len / VN;
#pragma unroll 4
      for (int v = lane; v < nvec; v += 32) {
        const uint4 xq = xv[v], gq = gv[v];
        const uint32_t xw[4] = {xq.x, xq.y, xq.z, xq.w};
        uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w};
        bool blocked = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (DT == kF32) {
            if (ir_element(__uint_as_float(xw[i]), __uint_as_float(gw[i]), ir, fast_mode, s)) {
              gw[i] = 0u;
              blocked = true;
            }
          } else {
            if (ir_element(__uint_as_float(xw[i] << 16), __uint_as_float(gw[i] << 16), ir, fast_mode, s)) {
              gw[i] &= 0xffff0000u;
              blocked = true;
            }
            if (ir_element(__uint_as_float(xw[i] & 0xffff0000u), __uint_as_float(gw[i] & 0xffff0000u), ir, fast_mode, s)) {
              gw[i] &= 0x0000ffffu;
              blocked = true;
            }
          }
        }
        if (blocked) gv[v] = make_uint4(gw[0], gw[1], gw[2], gw[3]);
      }
    } else {
      for (int i = lane; i < len; i += 32)
        if (ir_element(Elem<DT>::load(x, start + i), Elem<DT>::load(grad_x, start + i), ir, fast_mode, s))
          Elem<DT>::store(grad_x, start + i, 0.0f);
    }
    up += (double)s.up;
    down += (double)s.lo;
  }
  double cnt = (double)s.cnt;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    up += __shfl_xor_sync(0xffffffffu, up, o);
    down += __shfl_xor_sync(0xffffffffu, down, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) {
    part[warp][0] = up;
    part[warp][1] = down;
    part[warp][2] = cnt;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double sum = part[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < 8; ++w) sum += part[w][threadIdx.x];
    float* const p = partial + (((int64_t)t * gridDim.x + blockIdx.x) * 3 + threadIdx.x) * 2;
    const float high = (float)sum;
    p[0] = high;
    p[1] = isfinite(high) ? (float)(sum - (double)high) : 0.0f;  // an infinite sum stays infinite
  }
}

template <int DT>
__global__ void static_ir_final_kernel(const float* __restrict__ partial,
                                       const void* __restrict__ ir_used, int M, int n_partials, TileTable tt,
                                       float decay, float input_min_percentage,
                                       void* __restrict__ grad_ir, int fast_mode) {
  __shared__ double sm[3][256];
  int t = blockIdx.x;
  double a = 0.0, b = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < n_partials; i += blockDim.x) {
    const float* p = partial + ((int64_t)t * n_partials + i) * 6;
    a += (double)p[0] + (double)p[1];
    b += (double)p[2] + (double)p[3];
    c += (double)p[4] + (double)p[5];
  }
  sm[0][threadIdx.x] = a;
  sm[1][threadIdx.x] = b;
  sm[2][threadIdx.x] = c;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sm[0][threadIdx.x] += sm[0][threadIdx.x + o];
      sm[1][threadIdx.x] += sm[1][threadIdx.x + o];
      sm[2][threadIdx.x] += sm[2][threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    float ir = Elem<DT>::load(ir_used, t);
    float acc = rnd<DT>(fadd(0.0f, rnd<DT>((float)sm[0][0])));
    acc = rnd<DT>(fsub(acc, rnd<DT>((float)sm[1][0])));
    if (fast_mode) {
      Elem<DT>::store(grad_ir, t, acc);
      return;
    }
    acc = rnd<DT>(fmul(acc, ir));
    if (decay > 0.0f) {
      float numel = (float)((double)M * (double)(tt.hi(t) - tt.lo(t)));
      float pct = fsub(1.0f, fdiv((float)sm[2][0], numel));
      float flag = pct > input_min_percentage ? 1.0f : 0.0f;
      float term = rnd<DT>(fmul(rnd<DT>(fmul(decay, ir)), flag));
      acc = rnd<DT>(fadd(acc, term));
    }
    Elem<DT>::store(grad_ir, t, acc);
  }
}

// Backward of the learned per-channel weight range (`quant_utils.py:125-151`, learn_res branch).
// One warp per (channel, tile) segment.  grad_w arrives as the gradient of the clipped /
// discretised weights and leaves as the gradient of the weights themselves (zero outside the
// range); grad_clip[t, n] is the fp32 row sum of (-Q | +Q | round(q) - q) * grad_w * grad_scale
// (below, above, inside the range), rounded to the layer dtype, and divided by n_states when the
// range entered the quantiser as range / n_states.  The reference builds its indicator tensors in
// fp32, so products and the row sum are fp32; the order of the row sum is this warp's.
template <int DT>
__global__ void __launch_bounds__(256)
learn_clip_backward_kernel(const void* __restrict__ w, const void* __restrict__ clip,
                           const int32_t* __restrict__ all_gt1, int N, int K, TileTable tt, int discretize,
                           float n_states, double max_state_d, int no_rounding,
                           void* __restrict__ grad_w, void* __restrict__ grad_clip) {
  const unsigned seg = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (seg >= (unsigned)N * (unsigned)tt.T) return;
  const int n = (int)(seg / (unsigned)tt.T), t = (int)(seg - (unsigned)n * (unsigned)tt.T);
  const int lo = tt.lo(t), len = tt.hi(t) - lo;
  const int64_t start = (int64_t)n * K + lo;
  const float c = Elem<DT>::load(clip, (int64_t)t * N + n);
  float res;
  if (discretize) {
    const float arg = rnd<DT>(fdiv(c, n_states));
    res = all_gt1[t] ? rnd<DT>(fdiv(2.0f, arg)) : rnd<DT>(fmul(2.0f, arg));
  } else {
    res = all_gt1[t] ? rnd<DT>(fdiv(1.0f, c)) : c;
  }
  if (res == 0.0f) res = 1.0f;
  const float resc = res < kTiny ? kTiny : res;
  const float q_max = discretize ? (float)max_state_d : 1.0f;  // as a Python float in the products
  const float q_cmp = rnd<DT>(q_max);                  // as the layer dtype in the comparisons
  const bool skip = !discretize || no_rounding != 0;
  // 1 / sqrt(numel) without rounding, 2 * sqrt(max_state / numel) with it, evaluated in double
  // like the Python expression and then used as an fp32 scalar (`quant_utils.py:103-106`)
  const double numel = (double)N * (double)len;
  const float grad_scale = (float)(skip ? 1.0 / sqrt(numel) : 2.0 * sqrt(max_state_d / numel));
  float acc = 0.0f;
  for (int i = lane; i < len; i += 32) {
    const float wv = Elem<DT>::load(w, start + i);
    const float g = Elem<DT>::load(grad_w, start + i);
    const float q = rnd<DT>(fdiv(wv, resc));
    const bool small = q < -q_cmp, big = q > q_cmp;
    float a;
    if (small) a = -q_max;
    else if (big) a = q_max;
    else a = skip ? 0.0f : rnd<DT>(fadd(-q, rnd<DT>(frint(q))));
    acc = fadd(acc, fmul(fmul(a, g), grad_scale));
    if (small || big) Elem<DT>::store(grad_w, start + i, 0.0f);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc = fadd(acc, __shfl_xor_sync(0xffffffffu, acc, o));
  if (lane == 0) {
    float r = rnd<DT>(acc);
    if (discretize) r = rnd<DT>(fdiv(r, n_states));
    Elem<DT>::store(grad_clip, (int64_t)t * N + n, r);
  }
}

}  // namespace

int launch_learn_clip_backward(int dtype, const void* w, const void* clip, const int32_t* all_gt1, int N,
                               int K, const TileTable& tt, int discretize, float n_states, double max_state,
                               int no_rounding, void* grad_w, void* grad_clip, cudaStream_t s) {
  ProfScope prof(AL_K_CLIP, s);
  int64_t segs = (int64_t)N * tt.T;
  unsigned blocks = (unsigned)((segs + 7) / 8);
  if (dtype == AL_F32)
    learn_clip_backward_kernel<kF32><<<blocks, 256, 0, s>>>(w, clip, all_gt1, N, K, tt, discretize, n_states, max_state, no_rounding, grad_w, grad_clip);
  else
    learn_clip_backward_kernel<kBF16><<<blocks, 256, 0, s>>>(w, clip, all_gt1, N, K, tt, discretize, n_states, max_state, no_rounding, grad_w, grad_clip);
  return check_launch("learn_clip_backward");
}

template <int DT, bool SPLIT>
static void bias_grad_any(const void* g, int M, int N, bool vec, int cols, int splits, float* partial, void* grad_bias,
                          cudaStream_t s) {
  const dim3 grid((N + cols - 1) / cols, kBiasCluster * splits);
  auto kernel = cols == 16 ? (vec ? bias_grad_kernel<DT, 4, 16, true, SPLIT> : bias_grad_kernel<DT, 1, 16, true, SPLIT>)
                           : (vec ? bias_grad_kernel<DT, 4, 64, true, SPLIT> : bias_grad_kernel<DT, 1, 64, true, SPLIT>);
  if (!SPLIT && grid.x > kBiasWideGroups)
    kernel = vec ? bias_grad_kernel<DT, 4, 64, false, false> : bias_grad_kernel<DT, 1, 64, false, false>;
  kernel<<<grid, kBiasThreads, 0, s>>>(g, M, N, splits, partial, grad_bias);
  if (SPLIT) bias_sum_kernel<DT><<<(N + kBiasThreads - 1) / kBiasThreads, kBiasThreads, 0, s>>>(partial, splits, N, grad_bias);
}

int launch_bias_grad(int dtype, const void* g, int M, int N, void* grad_bias, float* scratch, int64_t scratch_floats,
                     cudaStream_t s) {
  const uintptr_t align = dtype == AL_F32 ? 16 : 8;
  const bool vec = N % 4 == 0 && reinterpret_cast<uintptr_t>(g) % align == 0;
  const int cols = N <= 16 ? 16 : 64, groups = (N + cols - 1) / cols;
  // a tall gradient of few columns: several clusters per column group, while a thread keeps a run; their sums meet in the
  // caller's scratch
  const int ahead = bias_ahead(vec ? 4 : 1, true);
  const int pass = kBiasThreads / (cols / (vec ? 4 : 1)) * kBiasCluster;  // rows a cluster reads at a time
  int splits = kBiasCtas / (kBiasCluster * groups);
  if (splits > kBiasMaxSplits) splits = kBiasMaxSplits;
  if (splits > M / (pass * ahead)) splits = M / (pass * ahead);
  if (M < pass * (kBiasSplitRows * (4 + groups) / 4) || scratch == nullptr || (int64_t)splits * N > scratch_floats) splits = 1;
  if (splits < 1) splits = 1;
  ProfScope prof(AL_K_BIAS_GRAD, s, splits > 1 ? 2 : 1);
  auto run = dtype == AL_F32 ? (splits > 1 ? bias_grad_any<kF32, true> : bias_grad_any<kF32, false>)
                             : (splits > 1 ? bias_grad_any<kBF16, true> : bias_grad_any<kBF16, false>);
  run(g, M, N, vec, cols, splits, scratch, grad_bias, s);
  return check_launch("bias_grad");
}

int launch_static_ir_backward(int dtype, const void* x, const void* ir_used, void* grad_x, int M,
                              int K, const TileTable& tt, float decay, float input_min_percentage,
                              void* grad_ir, float* scratch, int fast_mode, cudaStream_t s) {
  ProfScope prof(AL_K_IR_BACKWARD, s, grad_ir ? 2 : 1);
  // 32 rows per block; 8 (a row per warp) where that leaves SMs without a block
  const int block_rows = (int64_t)M * tt.T >= 32 * 4 * 148 ? 32 : 8;
  const int n_partials = (M + block_rows - 1) / block_rows;
  const dim3 grid(n_partials, tt.T);
  const int vn = dtype == AL_F32 ? 4 : 8;
  bool vec = reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(grad_x) % 16 == 0 && K % vn == 0;
  for (int t = 0; t < tt.T; ++t) vec = vec && tt.hi(t) % vn == 0;
#define AL_STATIC_IR(DT_)                                                                                             \
  do {                                                                                                                \
    if (vec) static_ir_partial_kernel<DT_, true><<<grid, 256, 0, s>>>(x, ir_used, grad_x, M, K, tt, scratch, fast_mode, block_rows); \
    else static_ir_partial_kernel<DT_, false><<<grid, 256, 0, s>>>(x, ir_used, grad_x, M, K, tt, scratch, fast_mode, block_rows);    \
    if (grad_ir)                                                                                                      \
      static_ir_final_kernel<DT_><<<tt.T, 256, 0, s>>>(scratch, ir_used, M, n_partials, tt, decay,                    \
                                                       input_min_percentage, grad_ir, fast_mode);                     \
  } while (0)
  if (dtype == AL_F32) AL_STATIC_IR(kF32);
  else AL_STATIC_IR(kBF16);
#undef AL_STATIC_IR
  return check_launch("static_ir_backward");
}

}  // namespace al
