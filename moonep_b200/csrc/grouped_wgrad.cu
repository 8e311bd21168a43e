// Weight gradients of every group on tcgen05 tensor cores (sm_100a): contraction over the rows of a group,
//
//   dW[g] (P x Q, fp32) (=, +=) L[rows of g, :P]^T  @  R[rows of g, :Q]
//
// The operands are taken as stored (L: [rows, P], R: [rows, Q]; tiles are staged MN-major, see make_smem_desc_mn) or
// transposed (Lt: [P, ld], Rt: [Q, ld], the row index contiguous, K-major tiles as in the forward kernel).  The K loop
// of a tile runs over the group's rows (k0 = first row of the group, any multiple of 16 rows long; the last 64-row
// block issues only the MMAs that lie inside the group).  The groups that have anything to do are listed once per CTA in
// shared memory (in group order, the same list in every CTA), so empty groups cost nothing.  Per group, flags[g]
// selects: 0 store (and store zeros if the group has no rows), 1 add to what is there, 2 store, leave the target alone
// if the group has no rows.  A null out_ptrs[g] skips the group; rows without a target are reported through the status
// block.
//
// A cluster of two CTAs computes a 256 x 256 tile (cta_group::2, as in grouped_gemm_pair.cu): 32 KB of operands per CTA and
// 64 rows.  The accumulator is dW^T: TMEM lanes (the M index, 128 per CTA) run along Q, columns along P, so the 32 lanes of
// a warp hold 32 neighbours of a row of dW and every store instruction of the epilogue fills one 128-byte line straight from
// registers.  Lanes along P instead cost four times the L1 cycles (a sector per lane), or a turn through shared memory, whose
// slots the MMAs need.  When P is an odd multiple of 128 the last tile has 128 columns that are computed from zeros and not
// stored.  Short groups and a few odd numbers of SMs take one CTA per 256 x 128 tile of the same kernel instead (48 KB per
// 64 rows; the last tile of an odd P is 128 x 128): moonep_wgrad_single_cta.
//
// Bound by the tensor pipe and the fp32 results together: a tile of 1024 rows is 16 K blocks of MMAs and 256 KB of output.
// 8 groups x 1024 rows, 2048 x 7168: 183 us (1315 TFLOP/s), adding to the old values 224; 16 groups x 512 rows, 1024 x 2048:
// 41.  With MMAs and loads issued under `lane == 0` instead of by an elected lane of a warp that stays together: 239, 253, 47
// (and single CTAs 256, 296, 53).  What an accumulator waits for before it is used again is only that TMEM has been read
// (mbar_arrive_cluster): with an arrive that also waits for the stores to reach L2, groups of 128 rows take 38.6 us instead of
// 32.2 (16 groups, 1024 x 2048).  (Lanes along P, 32-byte stores: 236, 369, 57.7; results through shared memory in 512-byte bulk
// stores: 242 and 50 in a training step, an SM takes 15 clocks per bulk store.)
//
// Every mbarrier wait is bounded; on expiry the role records a status word and leaves its loop (see
// grouped_gemm_pair.cu for how a pair is torn down).
//
// No counterpart in the reference, which has no GEMM.
#include "umma.cuh"

namespace moonep {

namespace {

constexpr int kThreads = 192;
constexpr int kTmemCols = 512;
constexpr unsigned kHalfBytes = 128 * BK * 2;  // 16 KB: 128 columns of L or R
// A CTA stages 128 columns of R and, as one of a pair, 128 of L, alone 256: 192 KB of operands either way.
template <bool kPair> constexpr int kStages = kPair ? 6 : 4;
template <bool kPair> constexpr unsigned kStageBytes = (kPair ? 2 : 3) * kHalfBytes;
constexpr size_t kSmemBytes = 12 * kHalfBytes + 1024;
constexpr int kWgradMaxGroups = 512;  // groups per launch (their work list lives in shared memory)

// The weights of a layer share a launch: its waves of tiles are filled by all of them, and one tail is left instead of three.
// Training step, us: S=64, H=1024, I=256, 6 experts 92.3 -> 80.8; S=500, I=512, 12 experts 142.2 -> 129.7; S=1500, H=4096,
// I=1024, 8 experts 458 -> 447.
constexpr int kWgradWeights = 3;

struct WgradWeight {
  float* const* out_ptrs;  // [G] device array
  int P, Q, p_tiles, q_tiles;
};
struct WgradMaps {  // of each weight's operands
  CUtensorMap l[kWgradWeights], r[kWgradWeights];
};
struct WgradArgs {
  WgradWeight w[kWgradWeights];
  int n_weights;
  const int* flags;        // [G]
  const int* cu_seqlens;   // [G] inclusive padded ends
  const int* pads;         // [G, 2] or null: first of the group's last rows that hold zeros, and how many, or 0
  int* status;
  unsigned long long timeout_ns;
  int G, rows_cap;
  int early;      // launched with expert_pdl: the next kernel's CTAs may come while this one runs
  int row_major;  // operands are L [rows, P] and R [rows, Q] as they are (MN-major tiles) instead of their transposes
};


struct WgradGroups {  // per listed group: which group, its first row, its rows, target and mode
  int n;
  short g[kWgradMaxGroups];
  int start[kWgradMaxGroups];
  int krows[kWgradMaxGroups];
  int flag[kWgradMaxGroups];
  float* out[kWgradWeights][kWgradMaxGroups];
};

// Warp-collective: list the groups with rows, and the empty ones whose target must be zeroed, in group order.
__device__ __forceinline__ void wgrad_list_groups(const WgradArgs& a, WgradGroups& sg, int lane) {
  int n = 0;
  for (int base = 0; base < a.G; base += 32) {
    const int g = base + lane;
    bool listed = false;
    int start = 0, end = 0, krows = 0, flag = 0;
    float* out[kWgradWeights] = {};
    bool any = false;
    if (g < a.G) {
      group_bounds(a.cu_seqlens, g, a.rows_cap, start, end);
      krows = end > start ? end - start : 0;
      flag = a.flags[g];
      // the K coordinate of a TMA copy must be a multiple of 8 elements and the MMAs take 16 rows at a time:
      // a group that does not start and end on a multiple of 16 is refused (reported as rows without a target)
      if (((start | end) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < kWgradWeights; ++i)
          if (i < a.n_weights) {
            out[i] = a.w[i].out_ptrs[g];
            any = any || out[i] != nullptr;
          }
      }
      if (a.pads != nullptr && krows > 0) {  // rows of zeros add nothing: up to the next multiple of 16
        const int n = a.pads[2 * g + 1], used = (a.pads[2 * g] - start + 15) & ~15;
        if (n > 0 && used > 0 && used < krows && a.pads[2 * g] + n == end) krows = used;
      }
      listed = krows > 0 || (any && flag == 0);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, listed);
    const int pos = n + __popc(mask & ((1u << lane) - 1u));
    if (listed && pos < kWgradMaxGroups) {
      sg.g[pos] = (short)g;
      sg.start[pos] = start;
      sg.krows[pos] = krows;
      sg.flag[pos] = flag;
#pragma unroll
      for (int i = 0; i < kWgradWeights; ++i) sg.out[i][pos] = out[i];
    }
    n += __popc(mask);
  }
  if (lane == 0) sg.n = min(n, kWgradMaxGroups);
}

struct WgradTile {
  int i, g, pb, qb, k0, krows, flag, P, Q;  // of weight i
  float* out;
};

__device__ __forceinline__ long long wgrad_tiles(const WgradArgs& a, const WgradGroups& sg) {
  long long n = 0;
#pragma unroll
  for (int i = 0; i < kWgradWeights; ++i)
    if (i < a.n_weights) n += (long long)sg.n * a.w[i].p_tiles * a.w[i].q_tiles;
  return n;
}

__device__ __forceinline__ WgradTile wgrad_tile(const WgradArgs& a, const WgradGroups& sg, long long t) {
  WgradTile w;
  w.i = 0;
  while (w.i + 1 < a.n_weights) {
    const long long n = (long long)sg.n * a.w[w.i].p_tiles * a.w[w.i].q_tiles;
    if (t < n) break;
    t -= n;
    ++w.i;
  }
  const int q_tiles = a.w[w.i].q_tiles, per_group = a.w[w.i].p_tiles * q_tiles;
  const int idx = (int)(t / per_group);
  const int rem = (int)(t % per_group);
  w.pb = rem / q_tiles;
  w.qb = rem % q_tiles;
  w.P = a.w[w.i].P;
  w.Q = a.w[w.i].Q;
  w.g = sg.g[idx];
  w.k0 = sg.start[idx];
  w.krows = sg.krows[idx];
  w.flag = sg.flag[idx];
  w.out = sg.out[w.i][idx];
  return w;
}

// 32 accumulator columns (rows of dW, ld apart) of this lane's column of dW: stored, or added to what is there.
__device__ __forceinline__ void put_cols(float* dst, long long ld, const unsigned (&v)[32], bool add) {
  if (add) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      asm volatile("red.global.add.f32 [%0], %1;" ::"l"(dst + j * ld), "f"(__uint_as_float(v[j])) : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      asm volatile("st.global.L1::no_allocate.b32 [%0], %1;" ::"l"(dst + j * ld), "r"(v[j]) : "memory");
  }
}

template <bool kPair>
__device__ __forceinline__ void wgrad_body(const WgradMaps& maps, const WgradArgs& a) {
  constexpr int kStages = moonep::kStages<kPair>;
  constexpr unsigned kStageBytes = moonep::kStageBytes<kPair>;
  extern __shared__ unsigned char s_raw[];
  __shared__ __align__(8) unsigned long long s_full[kStages], s_empty[kStages], s_tfull[2], s_tempty[2], s_done;
  __shared__ unsigned s_tmem_base;
  __shared__ WgradGroups s_groups;
  unsigned char* s_tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(s_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned rank = kPair ? cluster_ctarank() : 0;  // 0: leader (issues the MMAs), 1: its peer
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(s_full + s, 1);   // used in the leader: its own arrive.expect_tx; both CTAs' copies complete the bytes
      mbar_init(s_empty + s, 1);  // one commit of the leader's MMA lane, delivered to both CTAs
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_tfull + b, 1);   // one commit, delivered to both CTAs
      mbar_init(s_tempty + b, kPair ? 8 : 4);  // used in the leader: four epilogue warps of each CTA
    }
    mbar_init(&s_done, 1);
    fence_barrier_init();
  }
  // What the kernels before wrote is read from here on.  TMEM, which one of them may still be about to take, is taken
  // after it.
  griddep_wait();
  if (a.early) griddep_launch();
  if (warp == 1) {
    tmem_alloc(&s_tmem_base, kTmemCols);
    tmem_relinquish();
  }
  if (warp == 0) wgrad_list_groups(a, s_groups, lane);
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();  // the peer's barriers exist before anything is delivered to them
  tc_fence_after();
  const unsigned tmem_base = s_tmem_base;
  // both CTAs own their whole TMEM, so the accumulators start at column 0 in both
  const bool tmem_ok = (tmem_base & 0xFFFFu) == 0;
  if (!tmem_ok && threadIdx.x == 0) gemm_fail(a.status, 14, 9, (int)tmem_base, 0);
  const long long unit = kPair ? blockIdx.x >> 1 : blockIdx.x, nunits = kPair ? gridDim.x >> 1 : gridDim.x;
  const long long num_tiles = wgrad_tiles(a, s_groups);

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (tmem_ok) {
      int stage = 0;
      unsigned phase = 0;
      bool failed = false;
      for (long long t = unit; t < num_tiles && !failed; t += nunits) {
        const WgradTile w = wgrad_tile(a, s_groups, t);
        if (w.krows == 0 || w.out == nullptr) continue;
        const int kbs = (w.krows + BK - 1) / BK;
        const int q0 = w.qb * (kPair ? BN : 128) + (int)rank * 128;
        const int p0 = w.pb * BN + (int)rank * 128;               // of a pair's second CTA it may lie past P: zeros
        const CUtensorMap *tmap_l = &maps.l[w.i], *tmap_r = &maps.r[w.i];
        const int cols = kPair ? 128 : min(BN, w.P - w.pb * BN);  // columns of L that this CTA stages
        for (int kb = 0; kb < kbs; ++kb) {
          if (!mbar_wait_warp(s_empty + stage, phase ^ 1u, a.timeout_ns)) {
            if (lane == 0) gemm_fail(a.status, 14, 1, stage, kb);
            failed = true;
            break;
          }
          if (elect_one()) {
            unsigned char* st = s_tiles + (size_t)stage * kStageBytes;
            const int k = w.k0 + kb * BK;
            if constexpr (kPair) {
              if (rank == 0) mbar_expect_tx(s_full + stage, 2 * kStageBytes);
              const unsigned full_of_leader = mapa_u32(s_full + stage, 0);
              if (a.row_major) {
                tma_load_mn_pair(st, tmap_r, q0 / 64, k, full_of_leader);
                tma_load_mn_pair(st + kHalfBytes, tmap_l, p0 / 64, k, full_of_leader);
              } else {
                tma_load_2d_pair(st, tmap_r, k, q0, full_of_leader);
                tma_load_2d_pair(st + kHalfBytes, tmap_l, k, p0, full_of_leader);
              }
            } else {
              mbar_expect_tx(s_full + stage, kHalfBytes + (unsigned)cols * BK * 2);
              if (a.row_major) {
                tma_load_mn(st, tmap_r, q0 / 64, k, s_full + stage);
                for (int c = 0; c < cols / 128; ++c)
                  tma_load_mn(st + (1 + c) * kHalfBytes, tmap_l, p0 / 64 + 2 * c, k, s_full + stage);
              } else {
                tma_load_2d(st, tmap_r, k, q0, s_full + stage);
                for (int c = 0; c < cols / 128; ++c)
                  tma_load_2d(st + (1 + c) * kHalfBytes, tmap_l, k, p0 + 128 * c, s_full + stage);
              }
            }
          }
          __syncwarp();
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader only): the whole warp waits, one lane issues ----------------
    if (rank == 0 && tmem_ok) {
      constexpr int M = kPair ? 2 * BM : BM;
      const unsigned kstep = a.row_major ? kDescStepMn : kDescStepK;
      const unsigned idesc_full = make_idesc(M, BN, a.row_major != 0, a.row_major != 0);
      const unsigned idesc_half = make_idesc(M, 128, a.row_major != 0, a.row_major != 0);
      // descriptors of stage 0; those of another lie a stage's bytes further, in 16-byte units
      const unsigned long long adesc0 = a.row_major ? make_smem_desc_mn(s_tiles) : make_smem_desc(s_tiles);
      const unsigned long long bdesc0 = a.row_major ? make_smem_desc_mn(s_tiles + kHalfBytes) : make_smem_desc(s_tiles + kHalfBytes);
      int stage = 0;
      unsigned phase = 0;
      unsigned tphase[2] = {0, 0};
      int it = 0;
      bool failed = false;
      for (long long t = unit; t < num_tiles && !failed; t += nunits) {
        const WgradTile w = wgrad_tile(a, s_groups, t);
        if (w.krows == 0 || w.out == nullptr) continue;
        const int buf = it & 1;
        ++it;
        if (!mbar_wait_warp(s_tempty + buf, tphase[buf] ^ 1u, a.timeout_ns)) {
          if (lane == 0) gemm_fail(a.status, 14, 2, buf, it);
          break;
        }
        tphase[buf] ^= 1u;
        const unsigned d_tmem = tmem_base + (unsigned)(buf * BN);
        const int kbs = (w.krows + BK - 1) / BK;
        const unsigned idesc = !kPair && w.P - w.pb * BN < BN ? idesc_half : idesc_full;  // half: the last tile of an odd P
        for (int kb = 0; kb < kbs; ++kb) {
          if (!mbar_wait_warp(s_full + stage, phase, a.timeout_ns)) {
            if (lane == 0) gemm_fail(a.status, 14, 3, stage, kb);
            failed = true;
            break;
          }
          tc_fence_after();
          const unsigned long long off = (unsigned long long)(stage * (int)(kStageBytes >> 4));
          const unsigned long long adesc = adesc0 + off, bdesc = bdesc0 + off;
          const int left = w.krows - kb * BK;
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk) {
              if (kk * UMMA_K >= left) break;  // MMAs inside the group
              const unsigned long long ad = adesc + (unsigned long long)(kk * kstep), bd = bdesc + (unsigned long long)(kk * kstep);
              const unsigned add = (kb | kk) != 0 ? 1u : 0u;
              if (kPair) umma_bf16_pair(d_tmem, ad, bd, idesc, add); else umma_bf16(d_tmem, ad, bd, idesc, add);
            }
            if (kPair) umma_commit_pair(s_empty + stage, 3); else umma_commit(s_empty + stage);
          }
          __syncwarp();
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!failed && elect_one()) {
          if (kPair) umma_commit_pair(s_tfull + buf, 3); else umma_commit(s_tfull + buf);
        }
        __syncwarp();
      }
      // nothing may be torn down under a running MMA: wait for everything issued so far
      if (elect_one()) {
        if (kPair) umma_commit_pair(&s_done, 1); else umma_commit(&s_done);
      }
      __syncwarp();
      if (!mbar_wait_warp(&s_done, 0, a.timeout_ns) && lane == 0) gemm_fail(a.status, 14, 5, 0, 0);
    }
    __syncwarp();
  } else {
    // ---------------- epilogue (warps 2..5, both CTAs): one column of dW per thread ----------------
    const int q = warp & 3;
    const unsigned tempty_of_leader[2] = {mapa_u32(s_tempty + 0, 0), mapa_u32(s_tempty + 1, 0)};
    unsigned tphase[2] = {0, 0};
    int it = 0;
    for (long long t = unit; tmem_ok && t < num_tiles; t += nunits) {
      const WgradTile w = wgrad_tile(a, s_groups, t);
      const int flag = w.flag;
      if (w.out == nullptr) {
        if (w.krows != 0 && rank == 0 && q == 0 && lane == 0 && w.pb == 0 && w.qb == 0 && a.status != nullptr &&
            atomicCAS(a.status + MOONEP_ST_CODE, 0, MOONEP_STATUS_BAD_INDEX) == 0) {
          a.status[MOONEP_ST_KERNEL] = 14;
          a.status[MOONEP_ST_FAMILY] = 100;  // kind: rows of a group whose gradient has no target
          a.status[MOONEP_ST_PEER] = w.g;
          a.status[MOONEP_ST_EXPECT] = 0;
          a.status[MOONEP_ST_SEEN] = w.krows;
          __threadfence();
        }
        continue;
      }
      float* out = w.out + (long long)w.pb * BN * w.Q + w.qb * (kPair ? BN : 128) + (int)rank * 128 + q * 32 + lane;
      const int cols = min(BN, w.P - w.pb * BN);  // rows of dW in this tile: 256, or 128 in the last tile of an odd P
      if (w.krows == 0) {
        if (flag == 0)
          for (int c = 0; c < cols; ++c) out[(long long)c * w.Q] = 0.f;
        continue;
      }
      const int buf = it & 1;
      ++it;
      int got = 1;
      if (lane == 0) got = mbar_wait_cluster(s_tfull + buf, tphase[buf], a.timeout_ns) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) {
        if (lane == 0) gemm_fail(a.status, 14, 4, buf, it);
        break;
      }
      tphase[buf] ^= 1u;
      tc_fence_after();
      const unsigned taddr = tmem_base + ((unsigned)(q * 32) << 16) + (unsigned)(buf * BN);
      const bool add = flag == 1;
      unsigned v[32], u[32];
      tmem_ld32(taddr, v);
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 64) {  // the load of 32 columns overlaps the stores of the 32 before
        tmem_ld_wait();
        tmem_ld32(taddr + (unsigned)(c0 + 32), u);
        put_cols(out + (long long)c0 * w.Q, w.Q, v, add);
        tmem_ld_wait();
        if (c0 + 64 < cols) tmem_ld32(taddr + (unsigned)(c0 + 64), v);
        put_cols(out + (long long)(c0 + 32) * w.Q, w.Q, u, add);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_of_leader[buf]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();  // nobody delivers to, or computes on, a CTA that has left
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    grouped_wgrad_kernel(const __grid_constant__ WgradMaps maps, const __grid_constant__ WgradArgs a) {
  wgrad_body<true>(maps, a);
}

__global__ void __launch_bounds__(kThreads, 1)
    grouped_wgrad_single_kernel(const __grid_constant__ WgradMaps maps, const __grid_constant__ WgradArgs a) {
  wgrad_body<false>(maps, a);
}

}  // namespace

}  // namespace moonep

using namespace moonep;

static int launch_single(const WgradMaps& maps, WgradArgs& a, int num_sms, void* stream) {
  static int sms = -1;
  if (sms < 0) {
    if (int rc = check_cuda(cudaFuncSetAttribute(grouped_wgrad_single_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kSmemBytes),
                            "cudaFuncSetAttribute(grouped_wgrad_single_kernel)"))
      return rc;
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    sms = n;
  }
  for (int i = 0; i < a.n_weights; ++i) a.w[i].q_tiles = a.w[i].Q / 128;
  const int grid = num_sms > 0 ? imin(num_sms, sms) : sms;
  if (int rc = check_cuda(launch_maybe_pdl(grouped_wgrad_single_kernel, grid, kThreads, kSmemBytes, (cudaStream_t)stream,
                                           a.early != 0, maps, a),
                          "launch grouped_wgrad_single_kernel"))
    return rc;
  return check_launch("grouped_wgrad_single_kernel");
}

// One CTA per tile, or pairs: 1 or 0.  rows_per_group: rows of a group that has any, as far as the caller knows; adds: its
// results are added to what is there, which is twice the traffic of the epilogue, so that the line lies at longer groups.
// Short groups are epilogue: a CTA's results are half a pair's, and the tail wave is finer.  Single against pair, us (adding):
// 8 groups, 2048 x 7168: 256 rows 101 and 104 (203, 207), 272 rows 112 and 100 (203, 207), 512 rows 146 and 123 (201, 205), 640
// rows 167 and 143 (218, 204); 64 groups, 640 x 1024: 256 rows 47.1 and 48.2 (75.8, 77.8), 272 rows 53.2 and 49.2 (75.8, 77.8),
// 512 rows 65.5 and 60.4 (77.8, 82.9), 640 rows 75.8 and 67.6 (87.0, 84.0); 16 groups, 2048 x 4096: 256 rows 112 and 120 (226,
// 234), 512 rows 164 and 137 (225, 229), 640 rows 196 and 167 (251, 230).  A pair cannot use the last of an odd number of SMs,
// and not one alone: 3 SMs 971 and 1400 us, 9 SMs 332 and 361 (16 groups x 128 rows), from there on the pair's rate makes up
// for it.
static int wgrad_on_single_ctas(int rows_per_group, int num_sms, bool adds) {
  return rows_per_group <= (adds ? 512 : 256) || (num_sms < 10 && (num_sms & 1) != 0) ? 1 : 0;
}
extern "C" int moonep_wgrad_single_cta(int rows_per_group, int num_sms) { return wgrad_on_single_ctas(rows_per_group, num_sms, false); }
extern "C" int moonep_wgrad_single_cta_adding(int rows_per_group, int num_sms) {
  return wgrad_on_single_ctas(rows_per_group, num_sms, true);
}

static int launch_wgrad(const WgradMaps& maps, WgradArgs& a, int rows_per_group, int adds,
                        int num_sms, void* stream) {
  a.early = expert_pdl(num_sms) ? 1 : 0;
  for (int i = 0; i < a.n_weights; ++i) a.w[i].p_tiles = (a.w[i].P + BN - 1) / BN;  // a pair computes 128 columns that are not stored in the last tile of an odd P
  if (rows_per_group <= 0) rows_per_group = a.rows_cap / a.G;
  if (wgrad_on_single_ctas(rows_per_group, imax(0, num_sms), adds != 0)) return launch_single(maps, a, num_sms, stream);
  for (int i = 0; i < a.n_weights; ++i) a.w[i].q_tiles = a.w[i].Q / BN;
  static int max_pairs = -1;  // pairs of these CTAs the device runs at once
  if (max_pairs < 0)
    if (int rc = pairs_at_once(grouped_wgrad_kernel, kThreads, kSmemBytes, "grouped_wgrad_kernel", &max_pairs)) return rc;
  int pairs = max_pairs;
  if (num_sms > 0) pairs = imin(pairs, num_sms / 2);
  if (int rc = check_cuda(launch_maybe_pdl(grouped_wgrad_kernel, 2 * pairs, kThreads, kSmemBytes, (cudaStream_t)stream,
                                           a.early != 0, maps, a),
                          "launch grouped_wgrad_kernel"))
    return rc;
  return check_launch("grouped_wgrad_kernel");
}

// lt: [P, ld] bf16 = L^T, rt: [Q, ld] bf16 = R^T (ld elements per row, a multiple of 8; the column index is the
// row of the dispatched shard).  For every group g with rows [cu[g-1], cu[g]) (a multiple of 16 long):
// out_ptrs[g][P, Q] fp32 = or += L_g^T R_g according to flags[g] (see the kernel).  out_ptrs and flags are
// device arrays of G entries.  P % 128 == 0, Q % 256 == 0.  rows_per_group (0: rows_cap / G) and adds: see
// wgrad_on_single_ctas.
extern "C" int moonep_grouped_wgrad(const void* lt, const void* rt, long long ld, int P, int Q, const int* cu_seqlens,
                                    int G, void* const* out_ptrs, const int* flags, int rows_cap, int* status,
                                    long long timeout_ms, int rows_per_group, int adds, int num_sms, void* stream) {
  if (P <= 0 || Q <= 0 || P % BM != 0 || Q % BN != 0) {
    set_error("moonep_grouped_wgrad: P must be a multiple of 128 and Q a multiple of 256");
    return 1;
  }
  if (G < 1 || G > kWgradMaxGroups) {
    set_error("moonep_grouped_wgrad: at most " + std::to_string(kWgradMaxGroups) + " groups per launch");
    return 1;
  }
  if (ld <= 0 || ld % 8 != 0 || rows_cap > ld) {
    set_error("moonep_grouped_wgrad: ld must be a multiple of 8 and at least rows_cap");
    return 1;
  }
  WgradMaps maps;
  if (int rc = make_tmap(&maps.l[0], lt, (unsigned long long)P, (unsigned long long)ld, 128)) return rc;
  if (int rc = make_tmap(&maps.r[0], rt, (unsigned long long)Q, (unsigned long long)ld, 128)) return rc;
  WgradArgs a;
  a.w[0] = {(float* const*)out_ptrs, P, Q, 0, 0};
  a.n_weights = 1;
  a.flags = flags;
  a.cu_seqlens = cu_seqlens;
  a.pads = nullptr;
  a.status = status;
  a.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 10000) * 1000000ull;
  a.G = G;
  a.rows_cap = rows_cap;
  a.row_major = 0;
  return launch_wgrad(maps, a, rows_per_group, adds, num_sms, stream);
}

// The same with the operands as they are: l = L [rows, P] and r = R [rows, Q] bf16, rows ldl / ldr elements apart
// (multiples of 8), so that column slices of wider tensors can be passed.  No transposed copies are needed: the
// tiles are staged MN-major (see make_smem_desc_mn).  Up to three weights of the same groups of rows in one launch (those after
// the first may be absent: l null).  pads (optional): a plan's zero_fill_ranges, whose rows hold zeros.
extern "C" int moonep_grouped_wgrad_layer(const void* l0, long long ldl0, const void* r0, long long ldr0, int P0, int Q0, void* const* out0,
                                          const void* l1, long long ldl1, const void* r1, long long ldr1, int P1, int Q1, void* const* out1,
                                          const void* l2, long long ldl2, const void* r2, long long ldr2, int P2, int Q2, void* const* out2,
                                          int rows, const int* cu_seqlens, int G, const int* flags, int* status, long long timeout_ms,
                                          int rows_per_group, int adds, int num_sms, const int* pads, void* stream) {
  if (G < 1 || G > kWgradMaxGroups) {
    set_error("moonep_grouped_wgrad_layer: at most " + std::to_string(kWgradMaxGroups) + " groups per launch");
    return 1;
  }
  const struct {
    const void *l, *r;
    long long ldl, ldr;
    int P, Q;
    void* const* out;
  } ws[kWgradWeights] = {{l0, r0, ldl0, ldr0, P0, Q0, out0}, {l1, r1, ldl1, ldr1, P1, Q1, out1}, {l2, r2, ldl2, ldr2, P2, Q2, out2}};
  WgradMaps maps;
  WgradArgs a;
  a.n_weights = 0;
  for (const auto& w : ws) {
    if (w.l == nullptr && a.n_weights > 0) break;
    if (w.P <= 0 || w.Q <= 0 || w.P % BM != 0 || w.Q % BN != 0) {
      set_error("moonep_grouped_wgrad_layer: P must be a multiple of 128 and Q a multiple of 256");
      return 1;
    }
    if (w.ldl < w.P || w.ldr < w.Q || w.ldl % 8 != 0 || w.ldr % 8 != 0 || rows <= 0) {
      set_error("moonep_grouped_wgrad_layer: row strides must be multiples of 8 and at least the matrix width");
      return 1;
    }
    const int i = a.n_weights++;
    if (int rc = make_tmap_mn(&maps.l[i], w.l, (unsigned long long)rows, (unsigned long long)w.P, (unsigned long long)w.ldl)) return rc;
    if (int rc = make_tmap_mn(&maps.r[i], w.r, (unsigned long long)rows, (unsigned long long)w.Q, (unsigned long long)w.ldr)) return rc;
    a.w[i] = {(float* const*)w.out, w.P, w.Q, 0, 0};
  }
  a.flags = flags;
  a.cu_seqlens = cu_seqlens;
  a.status = status;
  a.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 10000) * 1000000ull;
  a.G = G;
  a.rows_cap = rows;
  a.row_major = 1;
  a.pads = pads;
  return launch_wgrad(maps, a, rows_per_group, adds, num_sms, stream);
}
