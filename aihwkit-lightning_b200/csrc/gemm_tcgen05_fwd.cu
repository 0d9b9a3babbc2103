// Forward GEMM of the analog linear path on the Blackwell tensor cores (sm_100a):
//   out[m,n] = sum_t stage_t( xq[m, tile t] . w_mod[n, tile t] ) + bias[n]
// Operands are brought into shared memory by TMA (cp.async.bulk.tensor, 128-byte swizzle),
// multiplied by tcgen05.mma with fp32 accumulators in tensor memory (TMEM) and drained by
// tcgen05.ld.  One persistent, warp-specialised kernel: the K loop is cut at the analog-tile
// boundaries; each analog tile accumulates into one of two TMEM accumulators, and while the
// tensor core works on tile t+1 sixteen epilogue warps run tile t's output stage (rounding,
// output noise, ADC quantisation, clamp, clamp-mask bits) and add it to a running sum.  Large
// problems run on CTA pairs (256 x 256 blocks, cta_group::2), small ones on single CTAs
// (128 x 128 blocks, or 128 x 64 and 128 x 32 where those fill more of the chip).
#include "tcgen05_common.cuh"

namespace al {

namespace {

// ---------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------
struct FwdTcParams {
  int32_t small_adc_codes;  // |ADC code| provably below 2^38: unguarded add-based rint is exact
  int32_t tile_w;      // width of every analog tile (all equal on this path)
  int32_t ksteps;      // ceil(tile_w / 64)
  int32_t num_mb, num_nb;
  int32_t a_rows;      // single CTAs: rows a copy of A brings (fewer than 128 when M is smaller; the others of the
                       // stage keep what was there: they only reach outputs of rows that do not exist)
  float inp_res;       // fp32 layers: the A operand holds integer DAC codes, the accumulator is scaled by the DAC step
  FwdEpilogueParams ep;
  NoiseKeys noise;     // output-noise stream of this call, prepared on the host
  void* out;
};

constexpr int kRagStageWords = 32 * 9;
constexpr int rag_stage_bytes(int bn) { return fwd_epi_warps(false, bn) * kRagStageWords * 4; }

// normals of elements idx .. idx + 15 of the output-noise stream (normal4's groups of four, any idx)
__device__ __forceinline__ void normals16(uint64_t seed, uint64_t offset, uint64_t idx, float z[16]) {
  float b[20];
  const int r = (int)(idx & 3);
#pragma unroll
  for (int q = 0; q < 4; ++q) normal4(seed, offset, 1u, (idx >> 2) + q, b + 4 * q);
  if (r != 0) {
    normal4(seed, offset, 1u, (idx >> 2) + 4, b + 16);
    if (r & 1) {
#pragma unroll
      for (int i = 0; i < 19; ++i) b[i] = b[i + 1];
    }
    if (r & 2) {
#pragma unroll
      for (int i = 0; i < 18; ++i) b[i] = b[i + 2];
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) z[i] = b[i];
}

// MODE >= 0: the output stage is fixed at compile time (bit 0 output noise from the internal
// generator, bit 1 ADC quantisation, bit 2 clamp; reference rounding, per-tile scalar scales,
// rounding on, small ADC codes; fp32 layers: modes 0 and 1 only).  MODE < 0: every switch is read at run time.
//
// PAIR: launched as clusters of two CTAs that share one tcgen05.mma.cta_group::2 of 256 x 256
// per k-step (an MMA that is 256 columns wide runs the tensor cores at their full rate, one of
// 128 columns does not).  CTA `rank` owns rows [256 mb + 128 rank, +128) of the block: it stages
// those rows of the inputs and 128 of the block's 256 weight rows, holds its 128 x 256 half of
// the accumulator and runs the output stage on it.  The two accumulator buffers fill the tensor
// memory, so the running sum over the analog tiles (bf16x2) lives in shared memory, which leaves
// five pipeline stages.  Only the packed bf16 output stage exists in this form (the host sends
// per-channel scales and fp32 rounding to single CTAs).  The leader (rank 0) issues the MMAs;
// `full` collects both CTAs' copies in the leader, `empty` and `acc_full` are signalled in both
// CTAs by the leader's multicast commits, `acc_empty` collects both CTAs' epilogue warps in the
// leader.
//
// fp32 layers run pairs with 256 x 128 blocks: two accumulators and the fp32 running sum (128 columns each) fit the
// tensor memory, and a CTA stages 32 KiB per k-step for both planes where a single one stages 48 for the same products.
// 4096^3 with output noise on eight tiles: 295 us on single CTAs, 275 us on pairs, 205 us with the output stage fixed
// at compile time (MODE); 178 us with one tile, where the MMAs are the bound.  One 256-column MMA over both planes
// side by side, with the running sum in shared memory, was slower (287 us; 180 us with one tile).
//
// IO: element type of the layer's tensors (input ranges, bias, replayed noise, per-channel scales,
// outputs).  RAG: the row pitch of the outputs is no multiple of 8 (single CTAs, run-time output stage only): the
// output noise is addressed element by element -- with the generator of the CUDA-core GEMM, so that a layer draws the
// same noise on either engine -- and the outputs leave through a staging buffer, two rows of 16 columns per store,
// because a thread's own 16 columns start at no particular alignment (1000 x 2500 x 1500 with noise and ADC: 361 us on
// the CUDA cores, 43 us here).  IO = fp32: the A operand holds the DAC codes as bf16 integers and the weights come as
// bf16 planes (fourth dimension of their tensor map) that are accumulated one after the other;
// the output stage multiplies the accumulator by the DAC step of its (row, tile) first.
//
// BN: columns of a single CTA's block (pick_blocks; 256 x 4096 x 4096 with ADC: 27 us in 64 blocks of 128 columns, 15.8 us
// in 128 of 64 issued by elected threads).  A copy of A brings no rows beyond M.
// CHUNK: tiles of more than 64 * kRagChunkSteps columns (a kernel of its own: as a run-time switch it cost the others
// registers).
template <int RD, int MODE, bool PAIR, int IO = kBF16, bool RAG = false, int BN = F_BN, bool CHUNK = false>
__global__ void __launch_bounds__(fwd_threads(PAIR, BN), 1)
fwd_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
              const FwdTcParams p) {
  constexpr int kPlanesB = IO == kF32 ? kPlanes : 1;           // planes of the weights per stage
  constexpr bool kSumSmem = PAIR && IO == kBF16;               // running sum in shared memory, else in tensor memory
  constexpr int kStages = kSumSmem ? FP_STAGES : fwd_stages(BN, kPlanesB);
  constexpr int kBRows = BN;                                   // weight rows this CTA stages
  constexpr int kPlaneBytes = kBRows * BK * 2;
  constexpr int kStageBytes = fwd_stage_bytes(BN, kPlanesB);
  constexpr int kEpiWarps = fwd_epi_warps(PAIR, BN);
  static_assert(!PAIR || BN == (IO == kBF16 ? 128 : 64), "CTA pairs: 256 x 256 blocks of bf16, 256 x 128 of fp32 layers");
  constexpr int kBlockRows = PAIR ? 2 * BM : BM;               // rows of the outputs per work item
  constexpr int kBN = PAIR ? 2 * BN : BN;                      // columns of the outputs per work item
  constexpr int kSumBytes = kSumSmem ? FP_SUM_BYTES : 0;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stage_base = align_1024(smem_raw);
  uint8_t* sum_base = stage_base + kStages * kStageBytes;      // PAIR: [128 rows][256 bf16], 16-byte chunks swizzled
  Barriers* bars = reinterpret_cast<Barriers*>(sum_base + kSumBytes);
  volatile uint32_t* abort_flag = &bars->abort_flag;
  static_assert(!RAG || (MODE < 0 && !PAIR && IO == kBF16), "ragged outputs: run-time output stage on single CTAs");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const FwdEpilogueParams& ep = p.ep;
  const int chunks = CHUNK ? (p.ksteps + kRagChunkSteps - 1) / kRagChunkSteps : 1;  // accumulators per analog tile
  const int T = ep.T;
  const int num_tiles = p.num_mb * p.num_nb;  // num_mb counts blocks of kBlockRows rows
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const bool leader = rank == 0;
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int n_workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int row_off = (int)rank * BM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], PAIR ? 2 * kEpiWarps : kEpiWarps);
    }
    mbar_init(&bars->mma_done, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    if (PAIR) tmem_alloc_pair(&bars->tmem_slot, kTmemCols);
    else tmem_alloc(&bars->tmem_slot, kTmemCols);
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_slot;

  if (warp == 0) {
    // ---- TMA producer ------------------------------------------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&map_a);
      tma_prefetch_desc(&map_b);
      uint32_t it = 0;
      bool ok = true;
      for (int tile = worker; tile < num_tiles && ok; tile += n_workers) {
        const int mb = tile / p.num_nb, nb = tile % p.num_nb;
        for (int t = 0; t < T && ok; ++t) {
          for (int ks = 0; ks < p.ksteps; ++ks, ++it) {
            const int s = it % kStages;
            const uint32_t ph = (it / kStages) & 1u;
            if (!mbar_wait(&bars->empty[s], ph ^ 1u, abort_flag)) {
              raise_error(kErrProducer, abort_flag);
              ok = false;
              break;
            }
            uint8_t* sa = stage_base + s * kStageBytes;
            if (PAIR) {
              // both CTAs' copies complete on the leader's barrier
              if (leader) mbar_expect_tx(&bars->full[s], 2 * kStageBytes);
              const uint32_t bar = mapa_u32(smem_u32(&bars->full[s]), 0);
              tma_load_3d_pair(sa, &map_a, bar, ks * BK, t, mb * kBlockRows + row_off);
              if (IO == kF32) {
#pragma unroll
                for (int plane = 0; plane < kPlanesB; ++plane)
                  tma_load_4d_pair(sa + F_A_BYTES + plane * kPlaneBytes, &map_b, bar, ks * BK, t,
                                   nb * kBN + (int)rank * kBRows, plane);
              } else {
                tma_load_3d_pair(sa + F_A_BYTES, &map_b, bar, ks * BK, t, nb * kBN + (int)rank * kBRows);
              }
            } else {
              mbar_expect_tx(&bars->full[s], (uint32_t)(p.a_rows * BK * 2 + kPlanesB * kPlaneBytes));
              tma_load_3d(sa, &map_a, &bars->full[s], ks * BK, t, mb * BM);
              if (IO == kF32) {
#pragma unroll
                for (int plane = 0; plane < kPlanesB; ++plane)
                  tma_load_4d(sa + F_A_BYTES + plane * kPlaneBytes, &map_b, &bars->full[s], ks * BK, t, nb * BN, plane);
              } else {
                tma_load_3d(sa + F_A_BYTES, &map_b, &bars->full[s], ks * BK, t, nb * BN);
              }
            }
          }
        }
      }
      // drain: the last copies issued must have landed before the CTA may exit (the leader's
      // barrier covers its peer's copies; both CTAs meet at the end of the kernel)
      if (leader) {
        const uint32_t n_back = it < (uint32_t)kStages ? it : (uint32_t)kStages;
        for (uint32_t j = it - n_back; j < it; ++j) {
          const int s = j % kStages;
          const uint32_t ph = (j / kStages) & 1u;
          uint64_t t0 = globaltimer_ns();
          while (!mbar_try(&bars->full[s], ph)) {
            if (globaltimer_ns() - t0 > wait_limit_ns()) {
              raise_error(kErrDrain, abort_flag);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer --------------------------------------------------------------------
    if (leader && elect_one()) {
      constexpr uint32_t idesc = make_idesc(kBlockRows, kBN, 0, 0);
      uint32_t it = 0, acc_it = 0;
      bool ok = true;
      const bool withhold = *(volatile uint32_t*)&g_tc_withhold_acc_signal != 0u;  // test aid, see its declaration
      for (int tile = worker; tile < num_tiles && ok; tile += n_workers) {
        for (int part = 0; part < T * chunks && ok; ++part, ++acc_it) {  // chunk part % chunks of an analog tile
          const int b = acc_it & 1u;
          const uint32_t aph = (acc_it >> 1) & 1u;
          if (!mbar_wait(&bars->acc_empty[b], aph ^ 1u, abort_flag)) {
            raise_error(kErrMma, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(b * kBN);
          const int ks0 = CHUNK ? part % chunks * kRagChunkSteps : 0;
          const int ks1 = CHUNK ? min(ks0 + kRagChunkSteps, p.ksteps) : p.ksteps;
          for (int ks = ks0; ks < ks1; ++ks, ++it) {
            const int s = it % kStages;
            const uint32_t ph = (it / kStages) & 1u;
            if (!mbar_wait(&bars->full[s], ph, abort_flag)) {
              raise_error(kErrMma, abort_flag);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(stage_base + s * kStageBytes);
            const uint64_t da = desc_k_major(sa), db = desc_k_major(sa + F_A_BYTES);
#pragma unroll
            for (int plane = 0; plane < kPlanesB; ++plane)  // fp32: both planes meet the codes staged once
#pragma unroll
              for (int k4 = 0; k4 < BK / 16; ++k4) {
                const uint64_t dbp = db + (uint64_t)(plane * (kPlaneBytes >> 4) + k4 * 2);
                const uint32_t acc = ((ks - ks0) | k4 | plane) != 0 ? 1u : 0u;
                if (PAIR) umma_bf16_pair(d_tmem, da + (uint64_t)(k4 * 2), dbp, idesc, acc);
                else umma_bf16(d_tmem, da + (uint64_t)(k4 * 2), dbp, idesc, acc);
              }
            if (PAIR) umma_commit_pair(&bars->empty[s], 3);  // frees the stage in both CTAs
            else umma_commit(&bars->empty[s]);
          }
          if (ok && !withhold) {
            if (PAIR) umma_commit_pair(&bars->acc_full[b], 3);
            else umma_commit(&bars->acc_full[b]);
          }
        }
      }
      // all MMAs issued by this thread must have retired before TMEM is freed
      if (PAIR) umma_commit_pair(&bars->mma_done, 1);
      else umma_commit(&bars->mma_done);
      uint64_t t0 = globaltimer_ns();
      while (!mbar_try(&bars->mma_done, 0)) {
        if (globaltimer_ns() - t0 > wait_limit_ns()) {
          raise_error(kErrDrain, abort_flag);
          break;
        }
      }
    }
  } else if (warp >= 4) {
    // ---- epilogue: per-tile output stage and running sum ----------------------------------
    // warp & 3 selects the TMEM lane quadrant (rows), (warp - 4) >> 2 the kCols columns
    constexpr int kCols = PAIR ? kBN / 4 : 32;
    const int quad = warp & 3;
    const int col0 = ((warp - 4) >> 2) * kCols;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    const int M = ep.M, N = ep.N;
    constexpr bool kFixed = MODE >= 0;
    const bool has_noise = kFixed ? (MODE & 1) != 0 : ep.has_noise != 0;
    const bool has_adc = kFixed ? (MODE & 2) != 0 : ep.has_adc != 0;
    const bool has_bound = kFixed ? (MODE & 4) != 0 : ep.has_bound != 0;
    const bool replay = kFixed ? false : ep.out_noise != nullptr;
    const bool no_round = kFixed ? false : ep.no_rounding != 0;
    const NoiseCounter noise_ctr = noise_counter(p.noise);
    const bool small_codes = kFixed ? true : p.small_adc_codes != 0;
    const bool per_channel = kFixed ? false : (ep.w_amax != nullptr && (ep.noise_pc || ep.bound_pc));
    // Output noise with nothing non-linear between the tiles (no ADC, no clamp): the T independent
    // Gaussian terms s_t * xi_t of an output add up to one Gaussian of variance sum_t s_t^2, so
    // one draw per output at the last tile replaces T draws -- same distribution up to the bf16
    // rounding of the partial sums, an eighth of the generator work on an 8-tile layer.  Replayed
    // noise (parity runs) never takes this route: it is applied tile by tile as given.
    constexpr bool kMergedNoise = kFixed && MODE == 1 && IO == kBF16;
    float noise_var = 0.0f;
    TileEpilogueCfg cfg;
    cfg.has_noise = ep.has_noise; cfg.has_bound = ep.has_bound; cfg.has_adc = ep.has_adc;
    cfg.no_rounding = ep.no_rounding; cfg.noise_coef = ep.noise_coef; cfg.out_bound = ep.out_bound;
    cfg.out_res = ep.out_res;
    uint32_t acc_it = 0;
    bool ok = true;
    for (int tile = worker; tile < num_tiles && ok; tile += n_workers) {
      const int mb = tile / p.num_nb, nb = tile % p.num_nb;
      const int m = mb * kBlockRows + row_off + quad * 32 + lane;
      const bool row_ok = m < M;
      const int n_first = nb * kBN + col0;
      for (int t = 0; t < T && ok; ++t, ++acc_it) {
        // all but the last chunk of a wide tile: added up in tensor memory
        for (int chunk = 0; CHUNK && chunk < chunks - 1 && ok; ++chunk, ++acc_it) {
          if (!mbar_wait(&bars->acc_full[acc_it & 1u], (acc_it >> 1) & 1u, abort_flag)) {
            if (lane == 0) raise_error(kErrEpilogue, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll 1
          for (int h = 0; h < kCols / 16; ++h) {
            uint32_t accr[16];
            const uint32_t partial = tmem_base + lane_base + (uint32_t)(3 * kBN + col0 + h * 16);
            tmem_ld16(tmem_base + lane_base + (acc_it & 1u) * (uint32_t)kBN + (uint32_t)(col0 + h * 16), accr);
            tmem_wait_ld();
            if (chunk > 0) add_tmem16(partial, accr);
            tmem_st16(partial, accr);
          }
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->acc_empty[acc_it & 1u]);
        }
        if (CHUNK && !ok) break;
        const int b = acc_it & 1u;
        const uint32_t aph = (acc_it >> 1) & 1u;
        // constants of this (row, analog tile): fetched and derived before waiting for the
        // accumulator, so that the load latency and the division overlap the tile's MMAs
        float ir = 0.0f;
        if (row_ok) {
          if (ep.ir_mode == AL_IR_DYNAMIC) ir = Elem<IO>::load(ep.ir_rows, (int64_t)t * M + m);
          else if (ep.ir_mode == AL_IR_STATIC) ir = Elem<IO>::load(ep.ir_rows, t);
        }
        const float t_max = ep.w_tile_max ? ep.w_tile_max[t] : 0.0f;
        // fp32 layers: accumulator = sum of code * weight; the DAC step turns it into the tile's product
        const float dac_step = IO == kF32 ? quant_step<kF32>(ir, p.inp_res) : 1.0f;
        float sc = rnd<RD>(fmul(t_max, rnd<RD>(fmul(ep.noise_coef, ir))));
        bool noise_now = has_noise;
        if (kMergedNoise) {
          noise_var = t == 0 ? sc * sc : fmaf(sc, sc, noise_var);
          noise_now = t == T - 1;
        } else {
          noise_var = sc * sc;
        }
        // fixed modes: the scale of the noise goes under the generator's square root
        const float noise_neg_c = kNegTwoLn2 * noise_var;
        const float bound = rnd<RD>(fmul(rnd<RD>(fmul(ir, ep.out_bound)), t_max));
        const float step = has_adc ? quant_step<RD>(bound, ep.out_res) : 1.0f;
        const float stepc = step < kTiny ? kTiny : step;
        const float rstep = __frcp_rn(stepc);
        if (!mbar_wait(&bars->acc_full[b], aph, abort_flag)) {
          if (lane == 0) raise_error(kErrEpilogue, abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t keep_bits = 0;
        // eight consecutive elements share one generator call (N is a multiple of 8 on this path)
        const uint64_t row_group8 = (((uint64_t)t * M + (row_ok ? m : 0)) * N) >> 3;
        const bool packed = RD == kBF16 && !per_channel;  // bf16x2 arithmetic, bf16x2 running sum
        const __nv_bfloat162 sc2 = __float2bfloat162_rn(sc), step2 = __float2bfloat162_rn(step);
        const __nv_bfloat162 bound2 = __float2bfloat162_rn(bound), nbound2 = __float2bfloat162_rn(-bound);
        const __nv_bfloat162 zero2 = __float2bfloat162_rn(0.0f);
        const uint64_t nstepc2 = f32x2_pack(-stepc, -stepc), rstep2 = f32x2_pack(rstep, rstep);
        const uint64_t magic2 = f32x2_pack(12582912.0f, 12582912.0f), nmagic2 = f32x2_pack(-12582912.0f, -12582912.0f);
        // fixed modes: ADC in packed bf16 arithmetic (stepc and its reciprocal are bf16 values or round to them)
        const __nv_bfloat162 y2 = __float2bfloat162_rn(rstep), nstepc2b = __float2bfloat162_rn(-stepc);
        // this thread's row of the shared-memory running sum (PAIR): chunk c of 8 columns sits at
        // 16 * (c ^ (row & 7)), so the eight rows a quarter-warp reads hit distinct banks
        const int srow = quad * 32 + lane;
        const uint32_t sum_row = smem_u32(sum_base) + (uint32_t)srow * (uint32_t)(kBN * 2);
        // word (t, first column of this warp / 32, row m) of the clamp mask; the next word of the row is M further
        uint32_t* const mask_p = ep.keep_mask != nullptr
                                     ? ep.keep_mask + ((int64_t)t * ep.mask_words + (n_first >> 5)) * M + (row_ok ? m : 0)
                                     : nullptr;
        // the compile-time output stages unroll the walk over this warp's columns: every offset below
        // becomes an immediate
        constexpr int kUnrollH = kFixed ? kCols / 16 : 1;
#pragma unroll kUnrollH
        for (int h = 0; h < kCols / 16; ++h) {
          const int cc = col0 + h * 16;
          const int nh = n_first + h * 16;
          const int n0 = n_first + (h >> 1) * 32;  // the 32 columns whose mask word this half belongs to
          // layers with few output channels: column groups beyond the last channel hold nothing (uniform
          // across the warp; a group is skipped as a whole, so that its mask word keeps its one writer)
          if (!kFixed && n0 >= N) break;
          if ((h & 1) == 0) keep_bits = 0;
          uint32_t accr[16], sumr[16];
          tmem_ld16(tmem_base + lane_base + (uint32_t)(b * kBN + cc), accr);
          if (t > 0) {
            if (kSumSmem) {
#pragma unroll
              for (int v = 0; v < 2; ++v) {
                const uint32_t addr = sum_row + (uint32_t)((((cc >> 3) + v) ^ (srow & 7)) << 4);
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(sumr[4 * v]), "=r"(sumr[4 * v + 1]), "=r"(sumr[4 * v + 2]), "=r"(sumr[4 * v + 3])
                             : "r"(addr) : "memory");
              }
            } else if (packed) {
              tmem_ld8(tmem_base + lane_base + (uint32_t)(2 * kBN + (cc >> 1)), sumr);
            } else {
              tmem_ld16(tmem_base + lane_base + (uint32_t)(2 * kBN + cc), sumr);
            }
          }
          tmem_wait_ld();
          if (CHUNK) add_tmem16(tmem_base + lane_base + (uint32_t)(3 * kBN + cc), accr);
          if (IO == kF32) {
#pragma unroll
            for (int j = 0; j < 16; ++j) accr[j] = __float_as_uint(fmul(__uint_as_float(accr[j]), dac_step));
          }
          if constexpr (kFixed && IO == kF32) {
            // ---- fp32 layer without ADC and clamp: noise and running sum --------------------------
            float z[16];
            if (has_noise) {
#pragma unroll
              for (int g8 = 0; g8 < 2; ++g8) {
                const int nq = nh + g8 * 8;
                normal8_keyed(p.noise, noise_ctr, row_group8 + (uint32_t)((nq < N ? nq : 0) >> 3), &z[g8 * 8]);
              }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float o = __uint_as_float(accr[j]);
              if (has_noise) o = fadd(o, fmul(sc, z[j]));
              sumr[j] = __float_as_uint(fadd(t == 0 ? 0.0f : __uint_as_float(sumr[j]), o));
            }
          } else if constexpr (kFixed) {
            // ---- output stage fixed at compile time: everything in packed bf16 arithmetic --------
            if (t == 0) {
#pragma unroll
              for (int pr = 0; pr < 8; ++pr) sumr[pr] = 0u;  // +0.0 in both halves
            }
            uint32_t kept = 0;  // bit 2*pr (low half) and bit 16 + 2*pr + 1 (high half): element kept
#pragma unroll
            for (int g8 = 0; g8 < 2; ++g8) {
              uint32_t bits[4];
              if (noise_now) {
                const int nq = nh + g8 * 8;
                philox7_keyed(p.noise, noise_ctr, row_group8 + (uint32_t)((nq < N ? nq : 0) >> 3), bits);
              }
#pragma unroll
              for (int q4 = 0; q4 < 4; ++q4) {
                const int pr = g8 * 4 + q4;  // element 2*pr in the low half, 2*pr+1 in the high half
                __nv_bfloat162 o2 = __floats2bfloat162_rn(__uint_as_float(accr[2 * pr]), __uint_as_float(accr[2 * pr + 1]));
                if (noise_now) o2 = box_muller16_fma(bits[q4], noise_neg_c, o2);
                if (has_adc) o2 = adc_bf16x2(o2, y2, nstepc2b, step2);
                if (has_bound) {
                  // kept <=> the clamp leaves the value unchanged (false for NaN, like the reference's
                  // -bound <= o <= bound)
                  const __nv_bfloat162 c2 = __hmin2_nan(__hmax2_nan(o2, nbound2), bound2);
                  kept |= __heq2_mask(c2, o2) & ((1u << (2 * pr)) | (1u << (17 + 2 * pr)));
                  o2 = c2;
                }
                sumr[pr] = as_u32(__hadd2_rn(as_bf162(sumr[pr]), o2));
              }
            }
            if (!has_bound) kept = 0xffffffffu;
            keep_bits |= ((kept | (kept >> 16)) & 0xffffu) << ((h & 1) * 16);
          } else {
          float z[16];
          if (RAG && noise_now) {
            normals16(ep.seed, ep.offset + (ep.offset_base != nullptr ? *ep.offset_base : 0ull),
                      ((uint64_t)t * M + (row_ok ? m : 0)) * N + nh, z);
          } else if (noise_now) {
#pragma unroll
            for (int g8 = 0; g8 < 2; ++g8) {
              const int nq = nh + g8 * 8;
              if (replay) {
                const uint64_t idx = ((uint64_t)t * M + (row_ok ? m : 0)) * N + (nq < N ? nq : 0);
                if (IO == kF32) {
                  const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(ep.out_noise) + idx);
                  const float4 lo4 = src[0], hi4 = src[1];
                  z[g8 * 8 + 0] = lo4.x; z[g8 * 8 + 1] = lo4.y; z[g8 * 8 + 2] = lo4.z; z[g8 * 8 + 3] = lo4.w;
                  z[g8 * 8 + 4] = hi4.x; z[g8 * 8 + 5] = hi4.y; z[g8 * 8 + 6] = hi4.z; z[g8 * 8 + 7] = hi4.w;
                } else {
                  const uint4 raw = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(ep.out_noise) + idx);
                  const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                  for (int q = 0; q < 4; ++q) {
                    z[g8 * 8 + 2 * q] = __uint_as_float(rw[q] << 16);
                    z[g8 * 8 + 2 * q + 1] = __uint_as_float(rw[q] & 0xffff0000u);
                  }
                }
              } else {
                normal8_keyed(p.noise, noise_ctr, row_group8 + (uint32_t)((nq < N ? nq : 0) >> 3), &z[g8 * 8]);
              }
            }
          }
          if (packed) {
            if (t == 0) {
#pragma unroll
              for (int pr = 0; pr < 8; ++pr) sumr[pr] = 0u;  // +0.0 in both halves
            }
            uint32_t kept = 0;  // bit 2*pr (low half) and bit 16 + 2*pr + 1 (high half): element kept
#pragma unroll
            for (int pr = 0; pr < 8; ++pr) {
              // element 2*pr in the low half, 2*pr+1 in the high half
              __nv_bfloat162 o2 = __floats2bfloat162_rn(__uint_as_float(accr[2 * pr]), __uint_as_float(accr[2 * pr + 1]));
              if (noise_now) {
                const __nv_bfloat162 z2 = __floats2bfloat162_rn(z[2 * pr], z[2 * pr + 1]);
                o2 = __hadd2_rn(o2, __hmul2_rn(sc2, z2));
              }
              if (has_adc) {
                // both elements of the pair side by side in fp32x2 arithmetic
                float q_lo, q_hi;
                f32x2_unpack(f32x2_div_rcp(f32x2_pack(__low2float(o2), __high2float(o2)), nstepc2, rstep2), &q_lo, &q_hi);
                const __nv_bfloat162 q2 = __floats2bfloat162_rn(q_lo, q_hi);
                float c_lo = __low2float(q2), c_hi = __high2float(q2);
                if (!no_round) {
                  // bf16-valued codes: the unguarded add-based rint is exact below 2^38
                  if (small_codes) {
                    f32x2_unpack(f32x2_add(f32x2_add(f32x2_pack(c_lo, c_hi), magic2), nmagic2), &c_lo, &c_hi);
                  } else {
                    c_lo = rint_magic(c_lo);
                    c_hi = rint_magic(c_hi);
                  }
                }
                // an integer-rounded bf16 value is a bf16 value: packing is a bit move
                const uint32_t c2 = __byte_perm(__float_as_uint(c_lo), __float_as_uint(c_hi), 0x7632);
                o2 = __hmul2_rn(as_bf162(c2), step2);
              }
              if (has_bound) {
                // kept <=> the clamp leaves the value unchanged (false for NaN, like the reference's
                // -bound <= o <= bound)
                const __nv_bfloat162 c2 = __hmin2_nan(__hmax2_nan(o2, nbound2), bound2);
                kept |= __heq2_mask(c2, o2) & ((1u << (2 * pr)) | (1u << (17 + 2 * pr)));
                o2 = c2;
              }
              sumr[pr] = as_u32(__hadd2_rn(as_bf162(sumr[pr]), o2));
            }
            if (!has_bound) kept = 0xffffffffu;
            keep_bits |= ((kept | (kept >> 16)) & 0xffffu) << ((h & 1) * 16);
          } else if (!per_channel) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float acc = __uint_as_float(accr[j]);
              float o = rnd_alu<RD>(acc);
              if (has_noise) o = rnd_alu<RD>(fadd(o, rnd_alu<RD>(fmul(sc, rnd_alu<RD>(z[j])))));
              bool keep = true;
              if (has_adc) {
                float code = rnd_alu<RD>(fdiv_rcp(o, stepc, rstep));
                if (!no_round) code = rint_magic(code);
                o = rnd_alu<RD>(fmul(code, step));
              }
              if (has_bound) {
                keep = fabsf(o) <= bound;
                o = fminf(fmaxf(o, -bound), bound);
              }
              float sum = t == 0 ? fadd(0.0f, o) : rnd_alu<RD>(fadd(__uint_as_float(sumr[j]), o));
              if (acc != acc) sum = acc;  // the integer rounding above does not preserve NaN
              sumr[j] = __float_as_uint(sum);
              keep_bits |= (keep ? 1u : 0u) << ((h & 1) * 16 + j);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int n = nh + j;
              const float cmax = n < N ? Elem<IO>::load(ep.w_amax, (int64_t)t * N + n) : 0.0f;
              bool keep;
              const float o = tile_epilogue<RD>(__uint_as_float(accr[j]), ir, ep.noise_pc ? cmax : t_max,
                                                ep.bound_pc ? cmax : t_max, has_noise ? rnd<RD>(z[j]) : 0.0f,
                                                cfg, &keep);
              sumr[j] = __float_as_uint(t == 0 ? fadd(0.0f, o) : rnd<RD>(fadd(__uint_as_float(sumr[j]), o)));
              keep_bits |= (keep ? 1u : 0u) << ((h & 1) * 16 + j);
            }
          }
          }  // !kFixed
          if (t < T - 1) {
            if (kSumSmem) {
#pragma unroll
              for (int v = 0; v < 2; ++v) {
                const uint32_t addr = sum_row + (uint32_t)((((cc >> 3) + v) ^ (srow & 7)) << 4);
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(sumr[4 * v]),
                             "r"(sumr[4 * v + 1]), "r"(sumr[4 * v + 2]), "r"(sumr[4 * v + 3]) : "memory");
              }
            } else if (packed) {
              tmem_st8(tmem_base + lane_base + (uint32_t)(2 * kBN + (cc >> 1)), sumr);
            } else {
              tmem_st16(tmem_base + lane_base + (uint32_t)(2 * kBN + cc), sumr);
            }
          } else if (RAG) {
            // final (ragged outputs): bias, convert, transpose through this warp's staging buffer
            uint32_t* const st = reinterpret_cast<uint32_t*>(bars + 1) + (warp - 4) * kRagStageWords;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float b0 = 0.0f, b1 = 0.0f;
              if (ep.bias) {
                if (nh + 2 * e < N) b0 = Elem<kBF16>::load(ep.bias, nh + 2 * e);
                if (nh + 2 * e + 1 < N) b1 = Elem<kBF16>::load(ep.bias, nh + 2 * e + 1);
              }
              uint32_t w;
              if (packed) {
                w = ep.bias ? as_u32(__hadd2_rn(as_bf162(sumr[e]), __floats2bfloat162_rn(b0, b1))) : sumr[e];
              } else {
                float f0 = __uint_as_float(sumr[2 * e]), f1 = __uint_as_float(sumr[2 * e + 1]);
                if (ep.bias) {
                  f0 = fadd(rnd<RD>(f0), b0);
                  f1 = fadd(rnd<RD>(f1), b1);
                }
                w = pack_bf16x2_rn(f0, f1);
              }
              st[lane * 9 + e] = w;  // nine words a row: the rows of a warp start on different banks
            }
            __syncwarp();
            const int m_first = mb * kBlockRows + quad * 32, col = lane & 15;
#pragma unroll 4
            for (int rr = lane >> 4; rr < 32; rr += 2)
              if (m_first + rr < M && nh + col < N)
                reinterpret_cast<uint16_t*>(p.out)[(int64_t)(m_first + rr) * N + nh + col] =
                    reinterpret_cast<const uint16_t*>(st + rr * 9)[col];
            __syncwarp();
          } else if (row_ok && IO == kF32) {
            // final (fp32 layer): bias, store 16 floats of this row
            float* dst = reinterpret_cast<float*>(p.out) + (int64_t)m * N + nh;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              if (nh + v * 4 < N) {
                float f[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  f[e] = __uint_as_float(sumr[v * 4 + e]);
                  if (ep.bias) f[e] = fadd(f[e], Elem<kF32>::load(ep.bias, nh + v * 4 + e));
                }
                *reinterpret_cast<float4*>(dst + v * 4) = make_float4(f[0], f[1], f[2], f[3]);
              }
            }
          } else if (row_ok) {
            // final: bias, convert, store 16 bf16 = 32 bytes of this row
            uint16_t* dst = reinterpret_cast<uint16_t*>(p.out) + (int64_t)m * N + nh;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              if (nh + v * 8 < N) {
                uint32_t w4[4];
                if (packed) {
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    __nv_bfloat162 s2 = as_bf162(sumr[v * 4 + e]);
                    if (ep.bias) {
                      const uint16_t* const pb = reinterpret_cast<const uint16_t*>(ep.bias) + nh + v * 8 + 2 * e;
                      const uint32_t b2 = (reinterpret_cast<uintptr_t>(ep.bias) & 2) == 0  // a view may start anywhere
                                              ? *reinterpret_cast<const uint32_t*>(pb)
                                              : (uint32_t)pb[0] | ((uint32_t)pb[1] << 16);
                      s2 = __hadd2_rn(s2, as_bf162(b2));
                    }
                    w4[e] = as_u32(s2);
                  }
                } else {
                  float f[8];
#pragma unroll
                  for (int e = 0; e < 8; ++e) {
                    f[e] = __uint_as_float(sumr[v * 8 + e]);
                    if (ep.bias) f[e] = fadd(rnd<RD>(f[e]), Elem<kBF16>::load(ep.bias, nh + v * 8 + e));
                  }
#pragma unroll
                  for (int e = 0; e < 4; ++e) w4[e] = pack_bf16x2_rn(f[2 * e], f[2 * e + 1]);
                }
                *reinterpret_cast<uint4*>(dst + v * 8) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
              }
            }
          }
          if ((h & 1) && mask_p != nullptr && row_ok && (n0 >> 5) < ep.mask_words)
            mask_p[(int64_t)(h >> 1) * M] = keep_bits;  // lanes = consecutive rows
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&bars->acc_empty[b]), 0));
          else mbar_arrive(&bars->acc_empty[b]);
        }
      }
    }
  }

  // (pairs) nothing of this CTA's shared or tensor memory may go while the peer can still signal
  // or use it: both CTAs meet before the tensor memory is released
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  tc_fence_after();
  if (warp == 1) {
    if (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace

bool tc_forward_supported(const AlDesc& d, const TileTable& tt) { return tc_shape_ok(d, tt); }

using FwdKernel = void (*)(const CUtensorMap, const CUtensorMap, const FwdTcParams);
template <bool PAIR, int BN = F_BN>
static FwdKernel pick_fwd_kernel(int mode, int round_dt) {
  switch (mode) {
    case 0: return fwd_tc_kernel<kBF16, 0, PAIR, kBF16, false, BN>;
    case 1: return fwd_tc_kernel<kBF16, 1, PAIR, kBF16, false, BN>;
    case 2: return fwd_tc_kernel<kBF16, 2, PAIR, kBF16, false, BN>;
    case 3: return fwd_tc_kernel<kBF16, 3, PAIR, kBF16, false, BN>;
    case 4: return fwd_tc_kernel<kBF16, 4, PAIR, kBF16, false, BN>;
    case 5: return fwd_tc_kernel<kBF16, 5, PAIR, kBF16, false, BN>;
    case 6: return fwd_tc_kernel<kBF16, 6, PAIR, kBF16, false, BN>;
    case 7: return fwd_tc_kernel<kBF16, 7, PAIR, kBF16, false, BN>;
    default:
      // CTA pairs exist for bf16 rounding only
      if (PAIR) return fwd_tc_kernel<kBF16, -1, PAIR>;
      return round_dt == AL_BF16 ? fwd_tc_kernel<kBF16, -1, false, kBF16, false, BN>
                                 : fwd_tc_kernel<kF32, -1, false, kBF16, false, BN>;
  }
}

// Columns of a single CTA's block (128, 64 or 32), or 0 when CTA pairs are the better choice
static int fwd_block_columns(int M, int N, int n_pairs = 0, int64_t pair_blocks = 0, int planes = 1) {
  return pick_blocks(n_pairs, pair_blocks, sm_count(), 128, 32,
                     [&](int bn) { return (int64_t)((M + BM - 1) / BM) * ((N + bn - 1) / bn); }, planes);
}

static int fwd_copy_rows(int M) { return M < BM ? (M + 7) / 8 * 8 : BM; }

static int small_adc_codes(int tile_w, const FwdEpilogueParams& ep) {
  // |o| <= tile_w * ir * wmax * (1 + noise) and step = 2 * out_bound * ir * wmax / states
  const double states = ep.out_res > 1.0f ? ep.out_res : (ep.out_res > 0.0f ? 1.0 / ep.out_res : 1.0);
  const double max_code = 8.0 * (double)tile_w * states / (2.0 * (ep.out_bound > 0.0f ? ep.out_bound : 1.0));
  return max_code < 274877906944.0 ? 1 : 0;  // 2^38
}

// how many CTA pairs of the forward kernel the device runs at once (0: it cannot)
static int max_fwd_pairs(FwdKernel kernel, int smem) {
  static FwdKernel seen[24];
  static int count[24];
  static int n_seen = 0;
  for (int i = 0; i < n_seen; ++i)
    if (seen[i] == kernel) return count[i];
  int clusters = 0;
  PairLaunch pl(2 * sm_count(), fwd_threads(true, F_BN), smem, nullptr);  // every pair kernel has that many threads
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &pl.cfg) != cudaSuccess) {
    cudaGetLastError();
    clusters = 0;
  }
  if (n_seen < 24) {
    seen[n_seen] = kernel;
    count[n_seen++] = clusters;
  }
  return clusters;
}

int launch_fwd_tc(int round_dt, const void* xq, const void* w_mod, int K, const TileTable& tt,
                  const FwdEpilogueParams& ep, int pairing, void* out, cudaStream_t s) {
  ProfScope prof(AL_K_FWD_GEMM, s);
  int w = 0;
  if (!uniform_tiles(tt, &w) || !aligned16(xq) || !aligned16(w_mod) || !aligned16(out)) {
    set_error("fwd_tc: operands must be 16-byte aligned with equally wide tiles");
    return AL_ERR_UNSUPPORTED;
  }
  FwdTcParams p;
  p.tile_w = w;
  p.ksteps = (w + BK - 1) / BK;
  p.num_mb = (ep.M + BM - 1) / BM;
  p.a_rows = fwd_copy_rows(ep.M);
  p.ep = ep;
  p.noise = make_noise_keys(ep.seed, ep.offset, 1u, ep.offset_base);
  p.out = out;
  p.inp_res = 0.0f;
  p.small_adc_codes = small_adc_codes(w, ep);
  const bool per_channel = ep.w_amax != nullptr && (ep.noise_pc || ep.bound_pc);
  // the compile-time output stages quantise in packed bf16 arithmetic, which needs every ADC code
  // beyond +-127 to end on the clamp (up to 254 states: the 8-bit converter and below)
  const bool fixed = round_dt == AL_BF16 && !per_channel && ep.out_noise == nullptr && !ep.no_rounding &&
                     p.small_adc_codes && (!ep.has_adc || adc_codes_fit_a_byte(ep.out_res, ep.has_bound != 0));
  const int mode = fixed ? ((ep.has_noise ? 1 : 0) | (ep.has_adc ? 2 : 0) | (ep.has_bound ? 4 : 0)) : -1;
  // CTA pairs (256 x 256 blocks, packed bf16 output stage only) or single CTAs: pick_blocks.
  // The runtime calls below also bind the device's primary context to the calling thread
  // (autograd runs backward on its own threads); the driver entry point that encodes the
  // tensor maps needs a current context.
  const bool pair_ok = pairing >= 0 && round_dt == AL_BF16 && !per_channel;
  const int pair_tiles = ((ep.M + 2 * BM - 1) / (2 * BM)) * ((ep.N + 2 * F_BN - 1) / (2 * F_BN));
  FwdKernel kernel = nullptr;
  int rc = AL_OK, pairs = 0;
  const int pair_smem = FP_SMEM;
  if (pair_ok) {
    kernel = pick_fwd_kernel<true>(mode, round_dt);
    rc = ensure_smem(kernel, pair_smem);
    if (rc) return rc;
    pairs = max_fwd_pairs(kernel, pair_smem);
  }
  const int columns = pairing > 0 && pairs > 0 ? 0 : fwd_block_columns(ep.M, ep.N, pairs, pair_tiles);
  const bool pair = columns == 0;
  const int bn = pair ? F_BN : columns;
  const int single_smem = fwd_smem(bn, 1);
  if (!pair) {
    kernel = bn == 128 ? pick_fwd_kernel<false, 128>(mode, round_dt)
             : bn == 64 ? pick_fwd_kernel<false, 64>(mode, round_dt) : pick_fwd_kernel<false, 32>(mode, round_dt);
    rc = ensure_smem(kernel, single_smem);
    if (rc) return rc;
    p.num_nb = (ep.N + bn - 1) / bn;
  } else {
    p.num_mb = (ep.M + 2 * BM - 1) / (2 * BM);
    p.a_rows = BM;
    p.num_nb = (ep.N + 2 * F_BN - 1) / (2 * F_BN);
  }
  CUtensorMap map_a, map_b;
  {
    uint64_t dims[3] = {(uint64_t)w, (uint64_t)tt.T, (uint64_t)ep.M};
    uint64_t strides[2] = {(uint64_t)w * 2, (uint64_t)K * 2};
    uint32_t box[3] = {BK, 1, (uint32_t)p.a_rows};
    rc = make_map(&map_a, xq, 3, dims, strides, box);
    if (rc) return rc;
  }
  {
    uint64_t dims[3] = {(uint64_t)w, (uint64_t)tt.T, (uint64_t)ep.N};
    uint64_t strides[2] = {(uint64_t)w * 2, (uint64_t)K * 2};
    uint32_t box[3] = {BK, 1, (uint32_t)bn};
    rc = make_map(&map_b, w_mod, 3, dims, strides, box);
    if (rc) return rc;
  }
  if (pair) {
    PairLaunch pl(2 * (pair_tiles < pairs ? pair_tiles : pairs), fwd_threads(true, F_BN), pair_smem, s);
    cudaError_t e = cudaLaunchKernelEx(&pl.cfg, kernel, map_a, map_b, p);
    if (e != cudaSuccess) {
      set_error("fwd_tc (pairs): %s", cudaGetErrorString(e));
      return AL_ERR_CUDA;
    }
    return check_launch("fwd_tc_pair");
  }
  int tiles = p.num_mb * p.num_nb;
  int grid = tiles < sm_count() ? tiles : sm_count();
  kernel<<<grid, fwd_threads(false, bn), single_smem, s>>>(map_a, map_b, p);
  return check_launch("fwd_tc");
}

// Ragged bf16 layers (tile widths, K or N no multiples of 8; operands in the pitched layout).  Measured on B200 against
// the CUDA-core kernels, device time of an evaluation and of forward + backward in us (CUDA cores -> here):
//   1000 x 2500 x 1500 train (tiles of 500)  1152 -> 122     1 x 1000 x 777      79 -> 25, 150 -> 54
//   333 x 1000 x 777 evaluation                99 -> 25     64 x 300 x 100       40 -> 20,  65 -> 49
//   16 x 4001 x 4001                          408 -> 66     32 x 70 x 70         25 -> 18,  42 -> 36
//   100 x 2000 x 20 (tiles of 20)            1039 -> 261    8000 x 100 x 10      36 -> 22, 125 -> 97
//   65536 x 1000 x 777                        4689 -> 351, 14007 -> 853
// so there is no lower size.  Three lines: tiles narrower than 8 columns would be mostly padding; tiles that are not as
// even as possible have no closed-form start (no module makes them); and beyond 8192 rows a layer with few products a
// row stays with the CUDA cores, which split the rows of a weight gradient over the chip where one CTA walks them all
// here (forward + backward: 32768 x 100 x 10 135 -> 193, 65536 x 147 x 64 309 -> 339, 65536 x 288 x 33 428 -> 424,
// 65536 x 500 x 100 1225 -> 574), and an evaluation with next to none (65536 x 27 x 16 56 -> 60, 65536 x 33 x 30 73 -> 63).
// Each tile is a block of its own here and a pass of its own there: the products count once per tile (65536 x 100 x 10
// in 5 tiles 448 -> 503, in 10 826 -> 688; 65536 x 300 x 30 in 38 3543 -> 1930).
bool tc_ragged_supported(const AlDesc& d, const TileTable& tt, RaggedTiles* rt) {
  if (d.dtype != AL_BF16 || (d.engine != AL_ENGINE_AUTO && d.engine != AL_ENGINE_PITCHED) || tc_tiling_ok(d, tt) ||
      !ragged_tiles(tt, rt))
    return false;
  const int64_t row_work = (int64_t)d.K * d.N * rt->T;
  if (rt->widest() < 8 || (d.M > 8192 && row_work < (d.save_for_backward ? 10000 : 500))) return false;
  return (int64_t)rt->T * rt->pitch < (1ll << 31);
}

template <int BN, bool CHUNK = false>
static FwdKernel pick_ragged_kernel(int round_dt) {
  return round_dt == AL_BF16 ? fwd_tc_kernel<kBF16, -1, false, kBF16, true, BN, CHUNK>
                             : fwd_tc_kernel<kF32, -1, false, kBF16, true, BN, CHUNK>;
}

int launch_fwd_tc_ragged(int round_dt, const void* xq, const void* w_mod, const RaggedTiles& rt,
                         const FwdEpilogueParams& ep, void* out, cudaStream_t s) {
  ProfScope prof(AL_K_FWD_GEMM, s);
  if (!aligned16(xq) || !aligned16(w_mod)) {
    set_error("fwd_tc_ragged: operands must be 16-byte aligned");
    return AL_ERR_UNSUPPORTED;
  }
  FwdTcParams p;
  p.tile_w = rt.widest();
  p.ksteps = (p.tile_w + BK - 1) / BK;
  p.num_mb = (ep.M + BM - 1) / BM;
  p.a_rows = fwd_copy_rows(ep.M);
  const bool chunked = p.ksteps > kRagChunkSteps;
  const int bn = chunked ? 64 : fwd_block_columns(ep.M, ep.N);
  p.num_nb = (ep.N + bn - 1) / bn;
  p.inp_res = 0.0f;
  p.ep = ep;
  p.noise = make_noise_keys(ep.seed, ep.offset, 1u, ep.offset_base);
  p.out = out;
  p.small_adc_codes = small_adc_codes(p.tile_w, ep);
  FwdKernel kernel = chunked     ? pick_ragged_kernel<64, true>(round_dt)
                     : bn == 128 ? pick_ragged_kernel<128>(round_dt)
                     : bn == 64  ? pick_ragged_kernel<64>(round_dt)
                                 : pick_ragged_kernel<32>(round_dt);
  const int smem = fwd_smem(bn, 1) + rag_stage_bytes(bn);
  int rc = ensure_smem(kernel, smem);
  if (rc) return rc;
  CUtensorMap map_a, map_b;
  const uint64_t row_bytes = (uint64_t)rt.T * rt.pitch * 2;
  for (int b = 0; b < 2; ++b) {
    uint64_t dims[3] = {(uint64_t)p.tile_w, (uint64_t)rt.T, (uint64_t)(b ? ep.N : ep.M)};
    uint64_t strides[2] = {(uint64_t)rt.pitch * 2, row_bytes};
    uint32_t box[3] = {BK, 1, (uint32_t)(b ? bn : p.a_rows)};
    rc = make_map(b ? &map_b : &map_a, b ? w_mod : xq, 3, dims, strides, box);
    if (rc) return rc;
  }
  const int tiles = p.num_mb * p.num_nb;
  kernel<<<tiles < sm_count() ? tiles : sm_count(), fwd_threads(false, bn), smem, s>>>(map_a, map_b, p);
  return check_launch("fwd_tc_ragged");
}

// fp32 with the DAC on and integer codes of at most 9 bits (exact in bf16), tiles as for bf16
bool tc_f32_supported(const AlDesc& d, const TileTable& tt) {
  if (d.dtype != AL_F32 || !tc_tiling_ok(d, tt)) return false;
  if (d.ir_mode == AL_IR_OFF || !(d.inp_res > 0) || d.no_rounding) return false;
  const double states = d.inp_res > 1.0 ? d.inp_res : 1.0 / d.inp_res;
  return states <= 510.0;
}

template <bool PAIR, int BN>
static FwdKernel pick_f32_kernel(int mode) {
  return mode == 0   ? fwd_tc_kernel<kF32, 0, PAIR, kF32, false, BN>
         : mode == 1 ? fwd_tc_kernel<kF32, 1, PAIR, kF32, false, BN>
                     : fwd_tc_kernel<kF32, -1, PAIR, kF32, false, BN>;
}

// Forward of an fp32 layer on the tensor cores: A = DAC codes as bf16 [M,K], B = the bf16 planes of the
// modified weights [kPlanes][N][K]; fp32 running sum in tensor memory.
int launch_fwd_tc_f32(const void* codes16, const void* w_planes, int K, const TileTable& tt,
                      const FwdEpilogueParams& ep, float inp_res, int pairing, void* out, cudaStream_t s) {
  ProfScope prof(AL_K_FWD_GEMM, s);
  int w = 0;
  if (!uniform_tiles(tt, &w) || !aligned16(codes16) || !aligned16(w_planes) || !aligned16(out)) {
    set_error("fwd_tc_f32: operands must be 16-byte aligned with equally wide tiles");
    return AL_ERR_UNSUPPORTED;
  }
  FwdTcParams p;
  p.tile_w = w;
  p.ksteps = (w + BK - 1) / BK;
  p.num_mb = (ep.M + BM - 1) / BM;
  p.a_rows = fwd_copy_rows(ep.M);
  const bool per_channel = ep.w_amax != nullptr && (ep.noise_pc || ep.bound_pc);
  const bool fixed = !ep.has_adc && !ep.has_bound && !per_channel && ep.out_noise == nullptr;
  const int mode = fixed ? (ep.has_noise ? 1 : 0) : -1;
  FwdKernel kernel = pick_f32_kernel<true, 64>(mode);
  int rc = ensure_smem(kernel, fwd_smem(64, kPlanes));
  if (rc) return rc;
  const int pairs = pairing >= 0 ? max_fwd_pairs(kernel, fwd_smem(64, kPlanes)) : 0;
  const int64_t pair_blocks = (int64_t)((ep.M + 2 * BM - 1) / (2 * BM)) * ((ep.N + BM - 1) / BM);
  const int columns = pairing > 0 && pairs > 0 ? 0 : fwd_block_columns(ep.M, ep.N, pairs, pair_blocks, kPlanes);
  const bool pair = columns == 0;
  const int bn = pair ? 64 : columns;  // weight rows a CTA stages
  p.num_nb = pair ? (ep.N + BM - 1) / BM : (ep.N + bn - 1) / bn;
  if (pair) {
    p.num_mb = (ep.M + 2 * BM - 1) / (2 * BM);
    p.a_rows = BM;
  }
  p.ep = ep;
  p.noise = make_noise_keys(ep.seed, ep.offset, 1u, ep.offset_base);
  p.out = out;
  p.inp_res = inp_res;
  p.small_adc_codes = 0;  // fp32 accumulators: guarded rint
  const int smem = fwd_smem(bn, kPlanes);
  if (!pair) {
    kernel = bn == 128  ? pick_f32_kernel<false, 128>(mode)
             : bn == 64 ? pick_f32_kernel<false, 64>(mode) : pick_f32_kernel<false, 32>(mode);
    rc = ensure_smem(kernel, smem);
    if (rc) return rc;
  }
  CUtensorMap map_a, map_b;
  {
    uint64_t dims[3] = {(uint64_t)w, (uint64_t)tt.T, (uint64_t)ep.M};
    uint64_t strides[2] = {(uint64_t)w * 2, (uint64_t)K * 2};
    uint32_t box[3] = {BK, 1, (uint32_t)p.a_rows};
    rc = make_map(&map_a, codes16, 3, dims, strides, box);
    if (rc) return rc;
  }
  {
    uint64_t dims[4] = {(uint64_t)w, (uint64_t)tt.T, (uint64_t)ep.N, (uint64_t)kPlanes};
    uint64_t strides[3] = {(uint64_t)w * 2, (uint64_t)K * 2, (uint64_t)ep.N * K * 2};
    uint32_t box[4] = {BK, 1, (uint32_t)bn, 1};
    rc = make_map(&map_b, w_planes, 4, dims, strides, box);
    if (rc) return rc;
  }
  const int tiles = p.num_mb * p.num_nb;
  if (pair) {
    PairLaunch pl(2 * (tiles < pairs ? tiles : pairs), fwd_threads(true, bn), smem, s);
    const cudaError_t e = cudaLaunchKernelEx(&pl.cfg, kernel, map_a, map_b, p);
    if (e != cudaSuccess) {
      set_error("fwd_tc_f32 (pairs): %s", cudaGetErrorString(e));
      return AL_ERR_CUDA;
    }
    return check_launch("fwd_tc_f32_pair");
  }
  const int grid = tiles < sm_count() ? tiles : sm_count();
  kernel<<<grid, fwd_threads(false, bn), smem, s>>>(map_a, map_b, p);
  return check_launch("fwd_tc_f32");
}

cudaError_t tc_fwd_take_error_word(uint32_t* code) { return take_error_word(code); }
cudaError_t tc_fwd_set_wait_limit(unsigned long long ns) { return set_wait_limit(ns); }
cudaError_t tc_fwd_set_withhold_acc_signal(uint32_t on) { return set_withhold_acc_signal(on); }

}  // namespace al
