// Forward path for a handful of rows (M <= 16, e.g. single-token decoding): the layer is bound by streaming the weights
// from HBM once, so one kernel reads every weight exactly once and takes from it both what the model needs of the
// weights -- the per-channel abs-max and the tile maximum -- and the tile dot products.  The per-tile output stage
// needs the tile maximum over ALL channels, which is known only when the whole tile has been streamed, so it runs in a
// second, tiny kernel over the [T, 16, N] fp32 partial results.
//
// Preconditions (checked by the caller): bf16, equally wide tiles with 16-byte aligned starts, no weight modifier active
// in this call (the GEMM reads `w` itself) and no output noise.
#include <cuda_bf16.h>

#include "tcgen05_common.cuh"

namespace al {

namespace {

constexpr int kRows = 16;  // columns of one MMA, rows of the layer's input; rows >= M are zero

// A resident CTA per SM walks the (128 channels, analog tile) items with eleven stages of 64 k in flight across item
// boundaries; the weights are the 128-row operand of tcgen05.mma and the quantised inputs its 16 columns, and eight
// warps read the same stage once more from shared memory for the abs-max of its channels.  A CTA per (64 channels,
// tile) with mma.sync, which staged (and quantised) its 16 KiB of inputs for 64 KiB of weights before its first product
// and left its last wave mostly empty, was slower at every size, calls replayed from a graph, in us (then -> now):
//   1 x 512 x 512 10.3 -> 8.1, 1 x 4096 x 4096 20.5 -> 15.4, 16 x 8192 x 3072 34.9 -> 25.5, 16 x 3072 x 16384 42.0 -> 31.8.
// Launched call by call the DAC pass in front costs a launch: a single row of 2048 x 2048 21.5 -> 24.1.
// Results differ from 64 bits by the same 1.664e-3 (bf16 outputs) as before.
constexpr int S_CH = 128;                                  // channels of an item: rows of the MMA
constexpr int S_W_BYTES = S_CH * BK * 2, S_X_BYTES = kRows * BK * 2;
constexpr int S_STAGE_BYTES = S_W_BYTES + S_X_BYTES;       // 18 KiB
constexpr int S_STAGES = 11;
constexpr int S_CONSUMERS = 256, S_THREADS = 128 + S_CONSUMERS;
constexpr int S_TMEM_COLS = 32;                            // two accumulators of 16 columns

struct StreamBarriers {
  uint64_t full[S_STAGES], empty[S_STAGES];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t mma_done;
  uint32_t tmem_slot, abort_flag;
  float amax[S_CH];
};
constexpr int S_SMEM = S_STAGES * S_STAGE_BYTES + (int)sizeof(StreamBarriers) + 1024;

struct StreamParams {
  int32_t M, N, T, ksteps, num_items;  // item i: channels [128 (i / T), +128) of tile i % T
  float* acc;                          // [T][16][N]
  uint16_t* w_amax;                    // [T][N]
  float* tile_max;                     // [T], zeroed by the caller
};

__global__ void __launch_bounds__(S_THREADS, 1)
smallm_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                     const StreamParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const stage_base = align_1024(smem_raw);
  StreamBarriers* const bars = reinterpret_cast<StreamBarriers*>(stage_base + S_STAGES * S_STAGE_BYTES);
  volatile uint32_t* const abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S_STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1 + S_CONSUMERS / 32);  // the MMAs' commit and the eight warps of the abs-max
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], 4);
    }
    mbar_init(&bars->mma_done, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&bars->tmem_slot, S_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_slot;

  if (warp == 0) {
    // ---- TMA producer --------------------------------------------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&map_w);
      tma_prefetch_desc(&map_x);
      uint32_t it = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < p.num_items && ok; item += gridDim.x) {
        const int nb = item / p.T, t = item - nb * p.T;
        for (int ks = 0; ks < p.ksteps; ++ks, ++it) {
          const int s = it % S_STAGES;
          if (!mbar_wait(&bars->empty[s], ((it / S_STAGES) & 1u) ^ 1u, abort_flag)) {
            raise_error(kErrProducer, abort_flag);
            ok = false;
            break;
          }
          uint8_t* const st = stage_base + s * S_STAGE_BYTES;
          mbar_expect_tx(&bars->full[s], S_STAGE_BYTES);
          tma_load_3d(st, &map_w, &bars->full[s], ks * BK, t, nb * S_CH);
          tma_load_3d(st + S_W_BYTES, &map_x, &bars->full[s], ks * BK, t, 0);
        }
      }
      const uint32_t n_back = it < (uint32_t)S_STAGES ? it : (uint32_t)S_STAGES;
      for (uint32_t j = it - n_back; j < it; ++j) {  // the last copies must have landed before the CTA exits
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try(&bars->full[j % S_STAGES], (j / S_STAGES) & 1u)) {
          if (globaltimer_ns() - t0 > wait_limit_ns()) {
            raise_error(kErrDrain, abort_flag);
            break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----------------------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(S_CH, kRows, 0, 0);
      uint32_t it = 0, acc_it = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < p.num_items && ok; item += gridDim.x, ++acc_it) {
        const int b = acc_it & 1u;
        if (!mbar_wait(&bars->acc_empty[b], ((acc_it >> 1) & 1u) ^ 1u, abort_flag)) {
          raise_error(kErrMma, abort_flag);
          break;
        }
        tc_fence_after();
        for (int ks = 0; ks < p.ksteps; ++ks, ++it) {
          const int s = it % S_STAGES;
          if (!mbar_wait(&bars->full[s], (it / S_STAGES) & 1u, abort_flag)) {
            raise_error(kErrMma, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t st = smem_u32(stage_base + s * S_STAGE_BYTES);
          const uint64_t dw = desc_k_major(st), dx = desc_k_major(st + S_W_BYTES);
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; ++k4)
            umma_bf16(tmem_base + (uint32_t)(b * kRows), dw + (uint64_t)(k4 * 2), dx + (uint64_t)(k4 * 2), idesc,
                      (ks | k4) != 0 ? 1u : 0u);
          umma_commit(&bars->empty[s]);
        }
        if (ok) umma_commit(&bars->acc_full[b]);
      }
      umma_commit(&bars->mma_done);  // retired before the tensor memory is freed
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try(&bars->mma_done, 0)) {
        if (globaltimer_ns() - t0 > wait_limit_ns()) {
          raise_error(kErrDrain, abort_flag);
          break;
        }
      }
    }
  } else if (warp >= 4) {
    // ---- abs-max of the channels (all eight warps), accumulators to memory (four of them per item, in turn) ------
    const int ct = threadIdx.x - 128, row = ct & (S_CH - 1), half = ct >> 7;  // half: 64 of a row's 128 bytes
    uint32_t it = 0, acc_it = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < p.num_items; item += gridDim.x, ++acc_it) {
      const int nb = item / p.T, t = item - nb * p.T;
      const int n = nb * S_CH + row;
      __nv_bfloat162 m2 = __float2bfloat162_rn(0.0f);
      for (int ks = 0; ks < p.ksteps && ok; ++ks, ++it) {
        const int s = it % S_STAGES;
        if (!mbar_wait(&bars->full[s], (it / S_STAGES) & 1u, abort_flag)) {
          if (lane == 0) raise_error(kErrTransform, abort_flag);
          ok = false;
          break;
        }
        const uint32_t row_addr = smem_u32(stage_base + s * S_STAGE_BYTES) + (uint32_t)row * 128u;
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // 16-byte chunk j of a row sits at j ^ (row & 7)
          uint32_t v[4];
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                       : "r"(row_addr + (uint32_t)(((half * 4 + c) ^ (row & 7)) << 4))
                       : "memory");
#pragma unroll
          for (int e = 0; e < 4; ++e) m2 = __hmax2(m2, __habs2(as_bf162(v[e])));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->empty[s]);
      }
      // the two halves of a row meet in the group whose turn it is to store this item
      const int b = acc_it & 1u;
      float amax = fmaxf(__low2float(m2), __high2float(m2));
      if (half != b) bars->amax[row] = amax;
      asm volatile("bar.sync 1, %0;" ::"n"(S_CONSUMERS) : "memory");
      if (half == b) {
        amax = fmaxf(amax, bars->amax[row]);
        if (ok && n < p.N) p.w_amax[(int64_t)t * p.N + n] = f32_to_bf16_bits(amax);
        float wmax = amax;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
        if (lane == 0 && ok) {
          unsigned int* const slot = reinterpret_cast<unsigned int*>(p.tile_max) + t;
          const unsigned int bits = __float_as_uint(wmax);
          if (bits > *reinterpret_cast<volatile unsigned int*>(slot)) atomicMax(slot, bits);
        }
        if (ok && !mbar_wait(&bars->acc_full[b], (acc_it >> 1) & 1u, abort_flag)) {
          if (lane == 0) raise_error(kErrEpilogue, abort_flag);
          ok = false;
        }
        if (ok) {
          tc_fence_after();
          uint32_t r[kRows];
          tmem_ld16(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(b * kRows), r);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->acc_empty[b]);
          if (n < p.N) {
            float* const dst = p.acc + (int64_t)t * kRows * p.N + n;
#pragma unroll
            for (int m = 0; m < kRows; ++m)
              if (m < p.M) dst[(int64_t)m * p.N] = __uint_as_float(r[m]);
          }
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(S_CONSUMERS) : "memory");  // amax[] may be written again
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, S_TMEM_COLS);
}

// out[m, n] = sum_t stage_t(acc[t, m, n]) + bias[n]; one thread per output
template <int RD>
__global__ void __launch_bounds__(256)
smallm_epilogue_kernel(const float* __restrict__ acc, FwdEpilogueParams ep, void* __restrict__ out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y;
  if (n >= ep.N) return;
  TileEpilogueCfg cfg;
  cfg.has_noise = 0; cfg.has_bound = ep.has_bound; cfg.has_adc = ep.has_adc;
  cfg.no_rounding = ep.no_rounding; cfg.noise_coef = ep.noise_coef; cfg.out_bound = ep.out_bound;
  cfg.out_res = ep.out_res;
  float sum = 0.0f;
  for (int t = 0; t < ep.T; ++t) {
    float ir = 0.0f;
    if (ep.ir_mode == AL_IR_DYNAMIC) ir = Elem<kBF16>::load(ep.ir_rows, (int64_t)t * ep.M + m);
    else if (ep.ir_mode == AL_IR_STATIC) ir = Elem<kBF16>::load(ep.ir_rows, t);
    const float t_max = rnd<kBF16>(ep.w_tile_max[t]);
    const float s_bound = ep.bound_pc ? Elem<kBF16>::load(ep.w_amax, (int64_t)t * ep.N + n) : t_max;
    bool keep;
    const float o = tile_epilogue<RD>(acc[((int64_t)t * kRows + m) * ep.N + n], ir, t_max, s_bound, 0.0f, cfg, &keep);
    sum = t == 0 ? fadd(0.0f, o) : rnd<RD>(fadd(sum, o));
  }
  if (ep.bias) sum = fadd(rnd<RD>(sum), Elem<kBF16>::load(ep.bias, n));
  Elem<kBF16>::store(out, (int64_t)m * ep.N + n, sum);
}

}  // namespace

int64_t smallm_scratch_floats(int N, int T) { return (int64_t)T * kRows * N; }

bool smallm_forward_supported(int M, int K, int N, const TileTable& tt) {
  if (M < 1 || M > kRows || K % 8 != 0 || N % 8 != 0) return false;
  int w = 0;
  return uniform_tiles(tt, &w) && w % 8 == 0;
}

int launch_fwd_smallm(int round_dt, const void* xq, const void* w, int K, const TileTable& tt,
                      const FwdEpilogueParams& ep, void* w_amax, float* tile_max, float* scratch, void* out,
                      cudaStream_t s, bool tile_max_zeroed) {
  ProfScope prof(AL_K_FWD_GEMM, s, 2);
  const int tile_w = tt.hi(0);
  int rc = ensure_smem(smallm_stream_kernel, S_SMEM);
  if (rc) return rc;
  cudaError_t e = tile_max_zeroed ? cudaSuccess : cudaMemsetAsync(tile_max, 0, sizeof(float) * tt.T, s);
  if (e != cudaSuccess) {
    set_error("fwd_smallm: %s", cudaGetErrorString(e));
    return AL_ERR_CUDA;
  }
  StreamParams p;
  p.M = ep.M; p.N = ep.N; p.T = tt.T;
  p.ksteps = (tile_w + BK - 1) / BK;
  p.num_items = (ep.N + S_CH - 1) / S_CH * tt.T;
  p.acc = scratch;
  p.w_amax = reinterpret_cast<uint16_t*>(w_amax);
  p.tile_max = tile_max;
  CUtensorMap map_w, map_x;
  for (int b = 0; b < 2; ++b) {
    uint64_t dims[3] = {(uint64_t)tile_w, (uint64_t)tt.T, (uint64_t)(b ? ep.M : ep.N)};
    uint64_t strides[2] = {(uint64_t)tile_w * 2, (uint64_t)K * 2};
    uint32_t box[3] = {BK, 1, (uint32_t)(b ? kRows : S_CH)};
    rc = make_map(b ? &map_x : &map_w, b ? xq : w, 3, dims, strides, box);
    if (rc) return rc;
  }
  smallm_stream_kernel<<<p.num_items < sm_count() ? p.num_items : sm_count(), S_THREADS, S_SMEM, s>>>(map_w, map_x, p);
  rc = check_launch("smallm_stream");
  if (rc) return rc;
  FwdEpilogueParams e2 = ep;
  e2.w_amax = w_amax;
  e2.w_tile_max = tile_max;
  dim3 grid2((ep.N + 255) / 256, ep.M);
  if (round_dt == AL_BF16) smallm_epilogue_kernel<kBF16><<<grid2, 256, 0, s>>>(scratch, e2, out);
  else smallm_epilogue_kernel<kF32><<<grid2, 256, 0, s>>>(scratch, e2, out);
  return check_launch("smallm_epilogue");
}

cudaError_t tc_small_take_error_word(uint32_t* code) { return take_error_word(code); }
cudaError_t tc_small_set_wait_limit(unsigned long long ns) { return set_wait_limit(ns); }

}  // namespace al
