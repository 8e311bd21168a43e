// Grouped expert GEMM for sm_100a: tcgen05 tensor cores, TMEM accumulators, TMA-fed shared memory.
//
//   Y[rows of group g, :] = X[rows of group g, :] @ W[g]^T        X: [rows, K] bf16, W: [G, N, K] bf16
//
// Groups are the padded row segments of a dispatched shard: cu_seqlens[g] is the inclusive end of
// group g and every non-empty segment is a multiple of 128 rows, so each 128-row block belongs to
// exactly one group.  The number of row blocks is read from cu_seqlens on the device; the host never
// synchronises.
//
// Persistent kernel, one CTA per SM, 320 threads:
//   warp 0      TMA producer: per 64-wide K block one 128x64 tile of X and two 128x64 tiles of W
//               (cp.async.bulk.tensor.2d, 128-byte swizzle, every CTA loads its own tiles) into a 4-stage ring; the
//               transaction bytes complete the stage's "full" mbarrier.
//   warp 1      allocates 512 TMEM columns (two 128x256 fp32 accumulators) and issues the MMAs from
//               one lane: four tcgen05.mma (M=128, N=256, K=16, bf16 -> fp32) per stage;
//               tcgen05.commit releases the stage and, after the last K block, publishes the
//               accumulator to the epilogue.
//   warps 2..9  epilogue: tcgen05.ld 32 columns at a time from their 32 TMEM lanes and their half of the
//               columns, apply the epilogue, convert to bf16, store.  While they drain one accumulator the
//               MMA warp fills the other.
// Epilogues: PLAIN  y = acc                                   (256 output columns per tile)
//            SWIGLU y = silu(acc[:, :128]) * acc[:, 128:]      (W tiles come from W_gate and W_up;
//                                                              128 output columns per tile)
//            SCALE  y = acc * row_scale[row]                   (down projection times the gate
//                                                              weight carried with the row)
// W may also be given as [G, K, N] (N contiguous, MN-major tiles; PLAIN only): the activation gradients, see
// moonep_grouped_gemm_kn.
// Every mbarrier wait is bounded; on expiry the role records a status word and leaves its loop, the
// CTA still frees its TMEM before it returns.
//
// The reference has no GEMM; this kernel serves the MoE-layer benchmark configuration (dispatch ->
// prefetch_weight -> grouped GEMM -> combine) named beside the reference's Buffer API
// (reference README.md:46-48).
#include <cstring>

#include "umma.cuh"

namespace moonep {

namespace {

constexpr int kStages = 4, kMaxStages = 8;
// A product of few row blocks has fewer tiles than there are SMs, and an SM that streams weights takes 48 KB per K block for a
// whole tile, 32 for one of half the columns and 24 for a quarter.  So tiles are halved, twice at most, as long as every part
// finds an SM of its own; the ring then has six or eight stages.  A layer's forward pass, us, whole tiles and parts: S=300, H=2048,
// I=512, 10 groups 48.4 and 44.1; S=100, H=4096, I=256, 4 groups 53.4 and 41.9; S=32, H=2048, I=2048, 8 groups 66.8 and 64.3.
// W comes in boxes of a quarter's rows for whole tiles too, which took the same time as boxes of 128.
constexpr int kMaxSplit = 4, kBoxRows = 128 / kMaxSplit;
// Two epilogue warps per quarter of the TMEM lanes: a decode step is one tile per CTA, whose epilogue nothing hides (SwiGLU of
// 16 groups x 128 rows, K=2048, N=1024: 38.2 us with one warp per quarter, 34.8 with two; K=512, N=256: 19.8 and 16.4).
constexpr int kEpilogueWarps = 8;
constexpr int kGemmThreads = 64 + 32 * kEpilogueWarps;
constexpr int kTmemCols = 512;
constexpr unsigned kATileBytes = BM * BK * 2;        // 16 KB
constexpr unsigned kBHalfBytes = 128 * BK * 2;       // 16 KB
constexpr unsigned kStageBytes = kATileBytes + 2 * kBHalfBytes;  // 48 KB, of a whole tile

struct GemmMaps {  // of X and of the weights' halves
  const CUtensorMap *a, *b0, *b1;
};
struct Ring {  // barriers: of the stages, and of the two accumulators
  unsigned long long full[kMaxStages], empty[kMaxStages], tfull[2], tempty[2];
};

template <int kSplit, bool kKn>
__device__ __forceinline__ void run_tiles(const GemmArgs& a, const GemmMaps& maps, unsigned char* s_tiles, Ring& ring, unsigned tmem_base,
                                          int row_blocks) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = a.n_tiles * kSplit;
  const long long num_tiles = (long long)row_blocks * n_tiles;
  const int b_rows_per_tile = ((a.mode == kSwiglu) ? 128 : 256) / kSplit;  // W rows consumed per output tile and tensor map
  constexpr int half_rows = 128 / kSplit;                                  // rows of either half of the W tile
  constexpr unsigned stage_bytes = kATileBytes + 2 * kBHalfBytes / kSplit;
  constexpr int stages = kSplit == 1 ? kStages : kSplit == 2 ? 6 : kMaxStages;  // 192 KB each
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    {
      int stage = 0;
      unsigned phase = 0;
      bool failed = false;
      auto load_weights = [&](unsigned char* st, int kb, int wslot, int nb) {
        if constexpr (kKn) {  // W is [slots, K, N], of one tensor or two
          const bool second = kb >= a.k_split;
          const int kdim = (second ? a.k_blocks - a.k_split : a.k_split) * BK;  // K rows per expert in that tensor
          const int y = wslot * kdim + (second ? kb - a.k_split : kb) * BK;
#pragma unroll
          for (int c = 0; c < 2 * half_rows / 64; ++c)
            tma_load_mn(st + c * 64 * BK * 2, second ? maps.b1 : maps.b0, nb * (2 * half_rows / 64) + c, y, ring.full + stage);
          return;
        }
        const int wrow0 = wslot * a.n_per_group + nb * b_rows_per_tile;
#pragma unroll
        for (int r = 0; r < half_rows; r += kBoxRows) {
          tma_load_2d(st + r * BK * 2, maps.b0, kb * BK, wrow0 + r, ring.full + stage);
          tma_load_2d(st + (half_rows + r) * BK * 2, a.mode == kSwiglu ? maps.b1 : maps.b0, kb * BK,
                      wrow0 + (a.mode == kSwiglu ? 0 : half_rows) + r, ring.full + stage);
        }
      };
      for (long long t = blockIdx.x; t < num_tiles && !failed; t += gridDim.x) {
        const int mb = (int)(t / n_tiles), nb = (int)(t % n_tiles);
        const int row0 = mb * BM;
        int lo = 0, hi = a.G - 1;  // first group whose end is beyond row0
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (a.cu_seqlens[mid] > row0) hi = mid; else lo = mid + 1;
        }
        int wslot = a.group_map != nullptr ? a.group_map[lo] : lo;
        if (wslot < 0 || wslot >= a.w_slots) {
          // a group whose weights this rank does not hold: reported, computed with slot 0 (in bounds), never trusted
          if (lane == 0) gemm_bad_index(a.status, 13, 13, lo, wslot);
          wslot = 0;
        }
        // A first tile's weights need not wait for the kernel that makes its rows, whose last CTAs leave memory and SMs idle: a
        // layer's pass, S=64, I=1024, 16 groups, H=2048 66.9 -> 64.8 us, H=4096 103.2 -> 100.3.
        int asked = 0;  // K blocks whose weights are on their way
        if (a.weights_early && t == blockIdx.x) {
          asked = min(stages, a.k_blocks);
          for (; stage < asked; ++stage) {
            if (elect_one()) {
              mbar_expect_tx(ring.full + stage, stage_bytes);
              load_weights(s_tiles + (size_t)stage * stage_bytes + kATileBytes, stage, wslot, nb);
            }
            __syncwarp();
          }
          stage = 0;
          griddep_wait();
        }
        for (int kb = 0; kb < a.k_blocks; ++kb) {
          if (!mbar_wait_warp(ring.empty + stage, phase ^ 1u, a.timeout_ns)) {
            if (lane == 0) gemm_fail(a.status, 13, 1, stage, kb);
            failed = true;
            break;
          }
          if (elect_one()) {
            unsigned char* st = s_tiles + (size_t)stage * stage_bytes;
            if (kb >= asked) mbar_expect_tx(ring.full + stage, stage_bytes);
            tma_load_2d(st, maps.a, kb * BK, row0, ring.full + stage);
            if (kb >= asked) load_weights(st + kATileBytes, kb, wslot, nb);
          }
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer: the whole warp waits, one lane issues ----------------
    {
      constexpr unsigned idesc = make_idesc(BM, BN / kSplit, false, kKn);
      constexpr unsigned bstep = kKn ? kDescStepMn : kDescStepK;
      // descriptors of stage 0; those of another lie a stage's bytes further, in 16-byte units
      const unsigned long long adesc0 = make_smem_desc(s_tiles);
      const unsigned long long bdesc0 = kKn ? make_smem_desc_mn(s_tiles + kATileBytes) : make_smem_desc(s_tiles + kATileBytes);
      int stage = 0;
      unsigned phase = 0;
      unsigned tphase[2] = {0, 0};
      int it = 0;
      bool failed = false;
      for (long long t = blockIdx.x; t < num_tiles && !failed; t += gridDim.x, ++it) {
        const int buf = it & 1;
        if (!mbar_wait_warp(ring.tempty + buf, tphase[buf] ^ 1u, a.timeout_ns)) {
          if (lane == 0) gemm_fail(a.status, 13, 2, buf, it);
          break;
        }
        tphase[buf] ^= 1u;
        const unsigned d_tmem = tmem_base + (unsigned)(buf * BN);
        for (int kb = 0; kb < a.k_blocks; ++kb) {
          if (!mbar_wait_warp(ring.full + stage, phase, a.timeout_ns)) {
            if (lane == 0) gemm_fail(a.status, 13, 3, stage, kb);
            failed = true;
            break;
          }
          tc_fence_after();
          const unsigned long long off = (unsigned long long)(stage * (int)(stage_bytes >> 4));
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk) {
              // 16 bf16 = 32 bytes further along K inside the swizzled 128-byte rows
              umma_bf16(d_tmem, adesc0 + off + (unsigned long long)(kk * kDescStepK), bdesc0 + off + (unsigned long long)(kk * bstep),
                        idesc, (kb | kk) != 0 ? 1u : 0u);
            }
            umma_commit(ring.empty + stage);
          }
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!failed && elect_one()) umma_commit(ring.tfull + buf);
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    const int q = warp & 3;            // TMEM lane quarter this warp may read
    const int half = (warp - 2) >> 2;  // which half of the columns is this warp's
    if (blockIdx.x == 0)  // while the first accumulator is being filled
      for (int g = threadIdx.x - 64; g < a.G; g += kGemmThreads - 64) gemm_check_end(a.status, 13, g, a.cu_seqlens[g]);
    unsigned tphase[2] = {0, 0};
    int it = 0;
    for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
      const int buf = it & 1;
      const int mb = (int)(t / n_tiles), nb = (int)(t % n_tiles);
      int got = 1;
      if (lane == 0) got = mbar_wait(ring.tfull + buf, tphase[buf], a.timeout_ns) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) {
        if (lane == 0) gemm_fail(a.status, 13, 4, buf, it);
        break;
      }
      tphase[buf] ^= 1u;
      tc_fence_after();
      const int row = mb * BM + q * 32 + lane;
      const unsigned taddr = tmem_base + ((unsigned)(q * 32) << 16) + (unsigned)(buf * BN);
      if (!kKn && a.mode == kSwiglu) {
        uint16_t* orow = a.out + (long long)row * a.ldo + (long long)nb * half_rows;
        // columns of a warp; of a quarter of a tile the second warps have none
        constexpr int mine = half_rows / 2 > 32 ? half_rows / 2 : 32;
#pragma unroll 1
        for (int c0 = half * mine; c0 < min(half_rows, half * mine + mine); c0 += 32) {
          unsigned g[32], u[32];
          tmem_ld32(taddr + (unsigned)c0, g);
          tmem_ld32(taddr + (unsigned)(half_rows + c0), u);
          tmem_ld_wait();
          unsigned o[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float y0 = silu(__uint_as_float(g[2 * j])) * __uint_as_float(u[2 * j]);
            const float y1 = silu(__uint_as_float(g[2 * j + 1])) * __uint_as_float(u[2 * j + 1]);
            o[j] = pack_bf16(y0, y1);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st16(orow + c0 + j * 8, make_int4((int)o[4 * j], (int)o[4 * j + 1], (int)o[4 * j + 2], (int)o[4 * j + 3]));
          if (a.pre_gate != nullptr) {
            const long long off = (long long)row * a.ldo + (long long)nb * half_rows + c0;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              g[j] = pack_bf16(__uint_as_float(g[2 * j]), __uint_as_float(g[2 * j + 1]));
              u[j] = pack_bf16(__uint_as_float(u[2 * j]), __uint_as_float(u[2 * j + 1]));
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              st16(a.pre_gate + off + j * 8, make_int4((int)g[4 * j], (int)g[4 * j + 1], (int)g[4 * j + 2], (int)g[4 * j + 3]));
              st16(a.pre_up + off + j * 8, make_int4((int)u[4 * j], (int)u[4 * j + 1], (int)u[4 * j + 2], (int)u[4 * j + 3]));
            }
          }
        }
      } else {
        const float scale = (a.mode == kScale && a.row_scale != nullptr) ? a.row_scale[row] : 1.f;
        uint16_t* orow = a.out + (long long)row * a.ldo + (long long)nb * 2 * half_rows;
#pragma unroll 1
        for (int c0 = half * half_rows; c0 < half * half_rows + half_rows; c0 += 32) {
          unsigned v[32];
          tmem_ld32(taddr + (unsigned)c0, v);
          tmem_ld_wait();
          unsigned o[16];
#pragma unroll
          for (int j = 0; j < 16; ++j)
            o[j] = pack_bf16(__uint_as_float(v[2 * j]) * scale, __uint_as_float(v[2 * j + 1]) * scale);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st16(orow + c0 + j * 8, make_int4((int)o[4 * j], (int)o[4 * j + 1], (int)o[4 * j + 2], (int)o[4 * j + 3]));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ring.tempty + buf);
    }
  }
}

template <bool kMaySplit, bool kKn>
__global__ void __launch_bounds__(kGemmThreads, 1)
    grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b0,
                        const __grid_constant__ CUtensorMap tmap_b1, const GemmArgs a) {
  extern __shared__ unsigned char s_raw[];
  __shared__ __align__(8) Ring ring;
  __shared__ unsigned s_tmem_base;
  unsigned char* s_tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(s_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(ring.full + s, 1);
      mbar_init(ring.empty + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(ring.tfull + b, 1);
      mbar_init(ring.tempty + b, kEpilogueWarps);
    }
    fence_barrier_init();
  }
  __syncthreads();  // the barriers exist
  unsigned tmem_base = 0;
  if (warp != 0) {
    // What the kernels before wrote is read from here on.  TMEM, which one of them may still be about to take, is taken
    // after it.
    griddep_wait();
    if (a.early) griddep_launch();
    if (warp == 1) {
      tmem_alloc(&s_tmem_base, kTmemCols);
      tmem_relinquish();
    }
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(kGemmThreads - 32) : "memory");
    tc_fence_after();
    tmem_base = s_tmem_base;
  } else if (!a.weights_early) {
    griddep_wait();
  }

  const int total_rows = min(a.cu_seqlens[a.G - 1], a.rows_cap);
  const int row_blocks = total_rows / BM;
  const GemmMaps maps = {&tmap_a, &tmap_b0, &tmap_b1};
  // a copy of the roles for each split: with sizes that are known only here, whole tiles took 0.7 us more per launch
  int split = 1;
  while (kMaySplit && split < kMaxSplit && (long long)row_blocks * a.n_tiles * split * 2 <= gridDim.x) split *= 2;
  if (split == 1)
    run_tiles<1, kKn>(a, maps, s_tiles, ring, tmem_base, row_blocks);
  else if (split == 2)
    run_tiles<2, kKn>(a, maps, s_tiles, ring, tmem_base, row_blocks);
  else
    run_tiles<kMaxSplit, kKn>(a, maps, s_tiles, ring, tmem_base, row_blocks);

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace

// ---- host side --------------------------------------------------------------------------------------

template <bool kMaySplit, bool kKn>
static int launch_of(const CUtensorMap& ta, const CUtensorMap& tb0, const CUtensorMap& tb1, const GemmArgs& a, int grid,
                     cudaStream_t stream) {
  const size_t smem = (size_t)kStages * kStageBytes + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    if (int rc = check_cuda(cudaFuncSetAttribute(grouped_gemm_kernel<kMaySplit, kKn>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem),
                            "cudaFuncSetAttribute(grouped_gemm_kernel)"))
      return rc;
    attr_set = true;
  }
  return check_cuda(launch_maybe_pdl(grouped_gemm_kernel<kMaySplit, kKn>, grid, kGemmThreads, smem, stream, a.early != 0, ta, tb0, tb1, a),
                    "launch grouped_gemm_kernel");
}

template <bool kKn>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb0, const CUtensorMap& tb1, GemmArgs& a, int num_sms, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = imax(1, num_sms > 0 ? imin(num_sms, sms) : sms);
  a.early = expert_pdl(num_sms) ? 1 : 0;
  // The rows are known on the device only.  Half the capacity stands for them here: a dispatched shard has room for almost two
  // blocks of padding per group.  The kernel that may cut tiles costs 0.4 us per launch where it does not (S=64, H=2048, I=1024,
  // 16 groups: a layer's pass 66.9 without and 67.9 with it).
  const bool may_split = (long long)a.rows_cap / BM * a.n_tiles <= grid;
  if (int rc = may_split ? launch_of<true, kKn>(ta, tb0, tb1, a, grid, stream)
                         : launch_of<false, kKn>(ta, tb0, tb1, a, grid, stream))
    return rc;
  return check_launch("grouped_gemm_kernel");
}

}  // namespace moonep

using namespace moonep;

// x: [rows_cap, K] bf16.  w0 (and w1 for SwiGLU): [G, n_per_group, K] bf16.  out: [rows_cap, n_out] bf16 with
// n_out = n_per_group (plain, scale) or n_per_group (swiglu: gate and up each have n_per_group rows).
// cu_seqlens: [G] int32 inclusive padded ends (multiples of 128).  mode: 0 plain, 1 swiglu, 2 scale by row_scale.
// group_map (optional): [G] int32, weight slot of every group when w holds only w_slots < G experts.
// pre_gate, pre_up (optional, SwiGLU): [rows_cap, n_per_group] bf16, receive x Wg^T and x Wu^T.
// weights_early: the kernel launched before on the stream writes none of w0, w1, cu_seqlens and group_map, and is no sooner
// done with waiting for its own predecessors than it lets this one start.
extern "C" int moonep_grouped_gemm(const void* x, const void* w0, const void* w1, void* out, const float* row_scale,
                                   const int* cu_seqlens, int G, int rows_cap, int K, int n_per_group, int mode,
                                   int* status, long long timeout_ms, int num_sms, const int* group_map, int w_slots,
                                   void* pre_gate, void* pre_up, int weights_early, void* stream) {
  if (group_map == nullptr || w_slots <= 0) w_slots = G;
  if ((pre_gate != nullptr) != (pre_up != nullptr) || (pre_gate != nullptr && mode != kSwiglu)) {
    set_error("moonep_grouped_gemm: pre_gate and pre_up go together and only with SwiGLU");
    return 1;
  }
  if (K % BK != 0 || K <= 0) {
    set_error("moonep_grouped_gemm: K must be a positive multiple of 64");
    return 1;
  }
  const int tile_n = (mode == kSwiglu) ? 128 : BN;
  if (n_per_group % tile_n != 0 || n_per_group <= 0) {
    set_error("moonep_grouped_gemm: N per group must be a multiple of " + std::to_string(tile_n));
    return 1;
  }
  if (mode == kSwiglu && w1 == nullptr) {
    set_error("moonep_grouped_gemm: SwiGLU needs the up-projection weights");
    return 1;
  }
  CUtensorMap ta, tb0, tb1;
  if (int rc = make_tmap(&ta, x, (unsigned long long)rows_cap, (unsigned long long)K, BM)) return rc;
  if (int rc = make_tmap(&tb0, w0, (unsigned long long)w_slots * n_per_group, (unsigned long long)K, kBoxRows)) return rc;
  tb1 = tb0;
  if (mode == kSwiglu)
    if (int rc = make_tmap(&tb1, w1, (unsigned long long)w_slots * n_per_group, (unsigned long long)K, kBoxRows)) return rc;
  GemmArgs a;
  a.out = (uint16_t*)out;
  a.row_scale = row_scale;
  a.cu_seqlens = cu_seqlens;
  a.status = status;
  a.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 10000) * 1000000ull;
  a.G = G;
  a.n_per_group = n_per_group;
  a.n_tiles = n_per_group / tile_n;
  a.k_blocks = K / BK;
  a.ldo = n_per_group;
  a.mode = mode;
  a.rows_cap = rows_cap;
  a.group_map = group_map;
  a.w_slots = w_slots;
  a.pre_gate = (uint16_t*)pre_gate;
  a.pre_up = (uint16_t*)pre_up;
  a.b_kn = 0;
  a.k_split = a.k_blocks;
  memset(&a.hooks, 0, sizeof(a.hooks));
  a.weights_early = weights_early;
  return launch<false>(ta, tb0, tb1, a, num_sms, (cudaStream_t)stream);
}

// The same with W given as [slots, K, N] (N contiguous), see moonep_grouped_gemm_pair_kn.  For groups of one row block, which
// leave the second CTA of a pair without rows: training step, us, on pairs and here: S=64, H=1024, I=256, 6 experts 80.7 and 71.0;
// S=500, I=512, 12 experts 129.6 and 117.2; S=200, H=2048, I=1024, 16 experts 339 and 323; S=1000 378 and 375.5.
extern "C" int moonep_grouped_gemm_kn(const void* x, const void* w0, int K0, const void* w1, int K1, void* out, const int* cu_seqlens,
                                      int G, int rows_cap, int N, int w_slots, int* status, long long timeout_ms, int num_sms,
                                      int weights_early, void* stream) {
  if (w1 == nullptr) K1 = 0;
  if (K0 <= 0 || K0 % BK != 0 || K1 < 0 || K1 % BK != 0 || N <= 0 || N % BN != 0 || w_slots <= 0) {
    set_error("moonep_grouped_gemm_kn: K0, K1 must be multiples of 64 and N a multiple of 256");
    return 1;
  }
  CUtensorMap ta, tb0, tb1;
  if (int rc = make_tmap(&ta, x, (unsigned long long)rows_cap, (unsigned long long)(K0 + K1), BM)) return rc;
  if (int rc = make_tmap_mn(&tb0, w0, (unsigned long long)w_slots * K0, (unsigned long long)N, 0, 1)) return rc;
  tb1 = tb0;
  if (K1)
    if (int rc = make_tmap_mn(&tb1, w1, (unsigned long long)w_slots * K1, (unsigned long long)N, 0, 1)) return rc;
  GemmArgs a;
  memset(&a, 0, sizeof(a));
  a.out = (uint16_t*)out;
  a.cu_seqlens = cu_seqlens;
  a.status = status;
  a.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 10000) * 1000000ull;
  a.G = G;
  a.n_per_group = N;
  a.n_tiles = N / BN;
  a.k_blocks = (K0 + K1) / BK;
  a.ldo = N;
  a.mode = kPlain;
  a.rows_cap = rows_cap;
  a.w_slots = w_slots;
  a.b_kn = 1;
  a.k_split = K0 / BK;
  a.weights_early = weights_early;
  return launch<true>(ta, tb0, tb1, a, num_sms, (cudaStream_t)stream);
}
