// Dispatch and combine of a Buffer with one rank, for sm_100a.
//
// With one rank nothing crosses a link and nothing is balanced: every routing entry lands on this GPU, the group
// layout is a prefix sum over the padded token counts, and the K entries of a token are one duplicate group.  The
// general kernels (dispatch.cu, combine_push.cu) reach that result through a chain of grid-wide hand-offs (publish,
// table stage on one CTA, token stage, link words walked by the expand role) which took 45 us of the 205 us of a
// dispatch at S=4096, H=7168, K=8, E=256 before most rows were written, and 65 of 84 us at S=16.  Here
//
//   dispatch   one launch whose CTAs wait for nobody.  Every CTA derives the whole group layout itself (E counts, one
//              prefix sum), starts clearing its share of the pad rows with asynchronous bulk stores, counts the
//              routing entries before its own contiguous range of tokens, gives its entries their rows, and streams
//              its tokens through shared memory: one bulk load and K bulk stores per piece of a row.  The pad rows'
//              stores (a third of the bytes at the size above) drain while the CTA plans.
//   combine    a warp per 512-byte piece of an output row, straight from the token's K destinations: no work counter,
//              no lists.
//
// Both are bound by HBM traffic: the rows are written (read) once, the tokens read (written) once.
//
// Parity: reference moonep_td/dispatch.py:42-117, moonep_td/_dedup_builder.py:23-108, moonep_td/combine.py:22-68 at one
// rank; the plan's contents are those of the general kernels (the order of the duplicate groups, which is arbitrary
// there, is token order here).
#include "common.cuh"
#include "host.h"

namespace moonep {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kCopyWarps = 8;     // warps that stream tokens, each through a ring of its own
constexpr int kRing = 3;          // pieces per ring: two loads run ahead of the stores
constexpr int kMaxPiece = 8192;   // bytes: 8 warps x 3 x 7 KB in flight at H=7168
constexpr int kEntries = 512;     // routing entries planned at a time (whole tokens)
constexpr int kPadGroups = 1024;  // groups whose pad rows are listed in shared memory at a time
constexpr int kMaxExperts = 4096; // three words of shared memory per expert
// Every CTA reads the routing before its own tokens: at 32 K entries that is 3 us for the last CTA, at 256 K about
// 25 us, where the general kernel's per-block histograms are the better way.
constexpr int kMaxEntries = 1 << 18;

struct SingleArgs {
  // planner (fresh plans)
  const int* topk;  // [N]
  const int* tpe;   // [E]
  int* dst;         // [N] written by a fresh dispatch, read by a replay
  int* cu_seqlens;
  int* experts_to_copy;
  int* zero_fill;  // [E+B, 2] written by a fresh dispatch, read by a replay
  int* remote_stats;
  int* dup_groups;
  int* dup_loffs;
  int* dup_counts;
  int* plan_src_info;  // [NvS] or null
  int* plan_link;      // [NvS] or null
  const uint16_t* hidden;  // [S, H]
  const float* weights;    // [S, K] or null
  int with_weights;        // pad rows' weight slots are cleared
  int fresh;
  int topk_vec;  // topk can be read 16 bytes at a time
  int vec_ok;    // rows can be moved 16 bytes at a time
  int bulk;      // rows go through shared memory with bulk copies
  int piece_bytes, npieces;
  int tokens_per_cta;
  int epoch_tpe, epoch_plan, epoch_sent;
};

struct SingleShared {
  unsigned long long bar[kCopyWarps * kRing];
  int warp_sum[kWarps];
  int pad_start[kPadGroups], pad_cum[kPadGroups];
  int loff[kEntries];  // destination row of every entry in hand, -1: none
  int bad;             // entries in hand without a row
};

// Inclusive prefix sum over the threads of the CTA; all threads call it.
__device__ __forceinline__ int block_scan(int v, int* warp_sum, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) warp_sum[warp] = v;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int x = warp_sum[w];
    if (w < warp) before += x;
    total += x;
  }
  __syncthreads();
  return v + before;
}

__device__ __forceinline__ int padded_rows(int cnt, int P) { return cnt > 0 ? ((cnt + P - 1) / P) * P : 0; }

// Visits this CTA's pad rows.  flag == false: clears them (bulk stores from `zeros`, not waited for) with their weights
// and, for a fresh plan, marks them unused in src_info and the plan's copies; flag == true: releases their row flags.
__device__ void visit_pads(const MoonepDevCtx& c, const SingleArgs& a, SingleShared& s, const int* cnt, const int* off,
                           const unsigned char* zeros, uint16_t* shard, int* meta, int epoch, bool flag) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = a.fresh ? c.E : c.E + c.B;  // the prefetch slots of a single rank are empty
  const long long row_bytes = (long long)c.H * 2;
  if (!a.fresh && a.zero_fill == nullptr) return;
  for (int g0 = 0; g0 < groups; g0 += kPadGroups) {
    const int n = min(kPadGroups, groups - g0);
    if (!flag || groups > kPadGroups) {  // one list only: the flag pass finds it as the first pass left it
      int carry = 0;
      for (int i0 = 0; i0 < n; i0 += kThreads) {
        const int i = i0 + threadIdx.x;
        int first = 0, rows = 0;
        if (i < n) {
          if (a.fresh) {
            const int k = cnt[g0 + i];
            first = off[g0 + i] + k;
            rows = k > 0 ? padded_rows(k, c.token_padding) - k : 0;
          } else {
            first = a.zero_fill[2 * (g0 + i)];
            rows = max(0, a.zero_fill[2 * (g0 + i) + 1]);
          }
        }
        int total;
        const int incl = block_scan(rows, s.warp_sum, total);
        if (i < n) {
          s.pad_start[i] = first;
          s.pad_cum[i] = carry + incl;
        }
        carry += total;
      }
      __syncthreads();
    }
    const int total = s.pad_cum[n - 1];
    auto row_of = [&](int j) {  // pad row j of the list, -1 when out of range
      int lo = 0, hi = n - 1;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (s.pad_cum[mid] > j) hi = mid; else lo = mid + 1;
      }
      const int row = s.pad_start[lo] + (j - (lo > 0 ? s.pad_cum[lo - 1] : 0));
      return row >= 0 && row < c.NvS ? row : -1;
    };
    // a thread per row; with bulk copies not a thread of the copy warps, whose rings would wait behind the clears
    const int first = a.bulk ? kCopyWarps * 32 : 0, nthr = kThreads - first;
    for (int j = blockIdx.x + gridDim.x * ((int)threadIdx.x - first); j >= 0 && j < total; j += gridDim.x * nthr) {
      const int row = row_of(j);
      if (row < 0) continue;
      if (flag) {
        st_relaxed_gpu(meta + c.rowflag_off + row, epoch);
        continue;
      }
      if (a.bulk) {
        unsigned char* p = reinterpret_cast<unsigned char*>(shard) + row * row_bytes;
        for (long long o = 0; o < row_bytes; o += a.piece_bytes)
          bulk_s2g(p + o, zeros, (unsigned)min((long long)a.piece_bytes, row_bytes - o));
      }
      if (a.with_weights) reinterpret_cast<float*>(meta + c.weights_off)[row] = 0.f;
      if (a.fresh) {
        meta[c.src_info_off + row] = -1;
        if (a.plan_src_info != nullptr) a.plan_src_info[row] = -1;
        if (a.plan_link != nullptr) a.plan_link[row] = 0;
      }
    }
    if (!flag) {
      if (a.bulk) {
        bulk_commit();
      } else {
        for (int j = blockIdx.x + gridDim.x * warp; j < total; j += gridDim.x * kWarps) {  // a warp per row
          const int row = row_of(j);
          if (row < 0) continue;
          uint16_t* p = shard + (long long)row * c.H;
          if (a.vec_ok) {
            for (int i = lane; i < c.H / 8; i += 32) st16(reinterpret_cast<int4*>(p) + i, make_int4(0, 0, 0, 0));
          } else {
            for (int i = lane; i < c.H; i += 32) p[i] = 0;
          }
        }
      }
    }
    __syncthreads();  // the lists are rewritten for the next groups
  }
}

// What one warp's ring holds.
struct Ring {
  unsigned char* stage;
  unsigned long long* bar;
  int loaded, stored;
};

// Copies the rows of `ntok` tokens (first: t0) to the rows in s.loff.  Pieces of rows are dealt to the copy warps; a
// lane per destination stores, so the K stores of a piece are issued together.  The last stores are left in flight.
__device__ bool copy_bulk(const MoonepDevCtx& c, const SingleArgs& a, const SingleShared& s, int t0, int ntok, Ring& r,
                          unsigned char* shard) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row_bytes = (long long)c.H * 2;
  const int items = ntok * a.npieces;
  const int mine = warp < items ? (items - warp + kCopyWarps - 1) / kCopyWarps : 0;
  auto load = [&](int n) {
    const int item = warp + n * kCopyWarps;
    const int tok = item / a.npieces, p = item - tok * a.npieces;
    const int q = r.loaded % kRing;
    if (lane == 0) {
      const long long o = (long long)p * a.piece_bytes;
      const unsigned len = (unsigned)min((long long)a.piece_bytes, row_bytes - o);
      mbar_expect_tx(r.bar + q, len);
      bulk_g2s(r.stage + (size_t)q * a.piece_bytes,
               reinterpret_cast<const unsigned char*>(a.hidden) + (t0 + tok) * row_bytes + o, len, r.bar + q);
    }
    ++r.loaded;
  };
  int ahead = 0;
  if (mine > 0) {
    bulk_wait_read<0>();  // every stage has been read by the stores of the tokens before
    __syncwarp();
    for (; ahead < min(mine, kRing - 1); ++ahead) load(ahead);
  }
  for (int n = 0; n < mine; ++n) {
    const int item = warp + n * kCopyWarps;
    const int tok = item / a.npieces, p = item - tok * a.npieces;
    const int loff = lane < c.K ? s.loff[tok * c.K + lane] : -1;
    const int q = r.stored % kRing;
    const bool got = mbar_wait(r.bar + q, (unsigned)((r.stored / kRing) & 1), c.timeout_ns);
    if (!__all_sync(0xffffffffu, got)) {
      if (lane == 0) record_status(c, MOONEP_STATUS_TIMEOUT, MOONEP_K_DISPATCH_EXPAND, 100, q, r.stored, t0 + tok);
      return false;
    }
    if (loff >= 0) {
      const long long o = (long long)p * a.piece_bytes;
      bulk_s2g(shard + loff * row_bytes + o, r.stage + (size_t)q * a.piece_bytes,
               (unsigned)min((long long)a.piece_bytes, row_bytes - o));
    }
    bulk_commit();
    ++r.stored;
    if (ahead < mine) {
      bulk_wait_read<1>();  // the stage to refill was stored from one item ago
      __syncwarp();
      load(ahead++);
    }
  }
  return true;
}

// The same without bulk copies: a warp per row, 16 bytes or one element at a time.
__device__ void copy_plain(const MoonepDevCtx& c, const SingleArgs& a, const SingleShared& s, int t0, int ntok,
                           uint16_t* shard) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int tok = warp; tok < ntok; tok += kWarps) {
    const uint16_t* src = a.hidden + (long long)(t0 + tok) * c.H;
    const int n = a.vec_ok ? c.H / 8 : c.H;
    for (int i = lane; i < n; i += 32) {
      if (a.vec_ok) {
        const int4 v = ld16(reinterpret_cast<const int4*>(src) + i);
        for (int k = 0; k < c.K; ++k) {
          const int loff = s.loff[tok * c.K + k];
          if (loff >= 0) st16(reinterpret_cast<int4*>(shard + (long long)loff * c.H) + i, v);
        }
      } else {
        const uint16_t v = src[i];
        for (int k = 0; k < c.K; ++k) {
          const int loff = s.loff[tok * c.K + k];
          if (loff >= 0) shard[(long long)loff * c.H + i] = v;
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1) dispatch_single_kernel(const MoonepDevCtx c, const SingleArgs a) {
  extern __shared__ __align__(128) unsigned char s_dyn[];  // rings, a piece of zeros, counts / offsets / cursors
  __shared__ __align__(8) SingleShared s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int E = c.E, K = c.K, NvS = c.NvS;
  unsigned char* zeros = s_dyn + (size_t)kCopyWarps * kRing * a.piece_bytes;
  int* cnt = reinterpret_cast<int*>(zeros + (a.bulk ? a.piece_bytes : 0));
  int* off = cnt + E;
  int* cur = off + E;
  if (tid < kCopyWarps * kRing) mbar_init(s.bar + tid, 1);
  if (a.bulk)
    for (int i = tid; i < a.piece_bytes / 16; i += kThreads) reinterpret_cast<int4*>(zeros)[i] = make_int4(0, 0, 0, 0);
  fence_barrier_init();
  fence_proxy_async();
  griddep_wait();
  griddep_launch();
  const unsigned long long t_begin = globaltimer_ns();
  // one answer for the CTA: the code below contains barriers
  const bool run = __syncthreads_and(poisoned(c) ? 0 : 1) != 0;
  bool ok = run;
  if (run) {
    int* meta = c.meta_peer[0];
    uint16_t* shard = c.hidden_peer[0];
    const int epoch = abs_epoch(c, MOONEP_FLAG_SENT, a.epoch_sent);
    int used = NvS;
    if (a.fresh) {
      int carry = 0;
      for (int e0 = 0; e0 < E; e0 += kThreads) {
        const int e = e0 + tid;
        const int n = e < E ? a.tpe[e] : 0;
        const int rows = padded_rows(n, c.token_padding);
        int total;
        const int end = carry + block_scan(rows, s.warp_sum, total);
        if (e < E) {
          cnt[e] = n;
          off[e] = end - rows;
          cur[e] = 0;
        }
        carry += total;
      }
      used = min(max(carry, 0), NvS);
      __syncthreads();
      if (blockIdx.x == 0) {
        for (int e = tid; e < E; e += kThreads) {
          const int n = cnt[e], rows = padded_rows(n, c.token_padding);
          a.cu_seqlens[e] = off[e] + rows;
          const bool pad = rows > n && n > 0;
          a.zero_fill[2 * e] = pad ? off[e] + n : 0;
          a.zero_fill[2 * e + 1] = pad ? rows - n : 0;
          meta[c.tpe_off + e] = n;
          c.tpe_prev[e] = 0;
          c.alloc_cum[e] = n;
          if (n > 0) c.expert_off[e] = off[e];
        }
        for (int b = tid; b < c.B; b += kThreads) {
          a.cu_seqlens[E + b] = carry;
          a.zero_fill[2 * (E + b)] = 0;
          a.zero_fill[2 * (E + b) + 1] = 0;
          a.experts_to_copy[b] = -1;
        }
        if (tid < 2) {
          a.remote_stats[tid] = 0;
          a.dup_counts[tid] = K > 1 ? (tid == 0 ? c.S : c.S * (K - 1)) : 0;
        }
        if (tid == 0 && carry > NvS) record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_PLAN_TABLES, 1, carry, NvS, 0);
        __syncthreads();
        if (tid == 0) {
          __threadfence();
          st_release_gpu(c.counters + MOONEP_CTR_TABLES_READY, abs_epoch(c, MOONEP_FLAG_PLAN, a.epoch_plan));
        }
      }
    }
    visit_pads(c, a, s, cnt, off, zeros, shard, meta, epoch, false);

    const int t_lo = min(c.S, (int)blockIdx.x * a.tokens_per_cta), t_hi = min(c.S, t_lo + a.tokens_per_cta);
    if (a.fresh) {
      for (int row = used + blockIdx.x * kThreads + tid; row < NvS; row += gridDim.x * kThreads) {
        meta[c.src_info_off + row] = -1;
        if (a.plan_src_info != nullptr) a.plan_src_info[row] = -1;
        if (a.plan_link != nullptr) a.plan_link[row] = 0;
      }
      if (t_lo < t_hi) {  // routing entries before this CTA's tokens
        const int n = t_lo * K;
        const int nv = a.topk_vec ? n / 4 : 0;
        auto count = [&](int e) {
          if ((unsigned)e < (unsigned)E) atomicAdd(cur + e, 1);
        };
        for (int i0 = tid; i0 < nv; i0 += 4 * kThreads) {
          int4 v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            v[u] = i0 + u * kThreads < nv ? __ldg(reinterpret_cast<const int4*>(a.topk) + i0 + u * kThreads)
                                          : make_int4(-1, -1, -1, -1);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            count(v[u].x);
            count(v[u].y);
            count(v[u].z);
            count(v[u].w);
          }
        }
        for (int i = nv * 4 + tid; i < n; i += kThreads) count(a.topk[i]);
      }
    }
    __syncthreads();

    Ring ring = {s_dyn + (size_t)warp * kRing * a.piece_bytes, s.bar + (warp < kCopyWarps ? warp : 0) * kRing, 0, 0};
    const int tokens_per_step = max(1, kEntries / K);
    float* wbuf = reinterpret_cast<float*>(meta + c.weights_off);
    for (int t0 = t_lo; t0 < t_hi; t0 += tokens_per_step) {
      const int ntok = min(tokens_per_step, t_hi - t0);
      const int nent = ntok * K, slot = t0 * K + tid;
      const bool in = tid < nent;
      int loff = -1;
      __syncthreads();  // the step before is done with s.loff and s.bad
      if (a.fresh) {
        int e = in ? a.topk[slot] : -1;
        if (in && (unsigned)e >= (unsigned)E) {
          record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_PLAN_TOKENS, 2, e, E, slot);
          e = -1;
        }
        if (tid == 0) s.bad = 0;
        // in-order index among the entries of the same expert: warp by warp, the warps before have moved the cursors on
        int idx = 0;
        for (int w = 0; w * 32 < nent; ++w) {
          if (warp == w) {
            const unsigned same = __match_any_sync(0xffffffffu, e >= 0 ? e : -1 - lane);
            if (e >= 0) idx = cur[e] + __popc(same & ((1u << lane) - 1u));
            __syncwarp();
            if (e >= 0 && lane == __ffs(same) - 1) cur[e] += __popc(same);
          }
          __syncthreads();
        }
        if (e >= 0) {
          if (idx >= cnt[e]) {
            record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_PLAN_TOKENS, 4, idx, e, slot);
          } else {
            loff = off[e] + idx;
            if (loff < 0 || loff >= NvS) {
              record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_PLAN_TOKENS, 3, loff, NvS, slot);
              loff = -1;
            }
          }
        }
        if (in && loff < 0) s.bad = 1;
      } else if (in) {
        const int d = a.dst[slot];
        loff = d < 0 ? -d - 1 : d;
        if (loff < 0 || loff >= NvS) {
          record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_DISPATCH_SEND, 6, d, slot / K, slot % K);
          loff = -1;
        }
      }
      if (in) s.loff[tid] = loff;
      __syncthreads();
      if (a.fresh && in) {
        const int k = tid % K, base = tid - k, tok = slot / K;
        // all entries of a token land on this rank: the first is its primary row, the others its duplicates in order
        int prev = k - 1, next = k + 1;
        if (s.bad) {  // some entry has no row (recorded above): skip such entries
          while (prev >= 0 && s.loff[base + prev] < 0) --prev;
          while (next < K && s.loff[base + next] < 0) ++next;
        }
        if (K > 1 && k == 0) {
          int first = s.loff[base], n = K - 1;
          if (s.bad) {
            first = -1, n = -1;
            for (int q = 0; q < K; ++q) {
              const int l = s.loff[base + q];
              if (l < 0) continue;
              if (n >= 0) a.dup_loffs[tok * (K - 1) + n] = l; else first = l;
              ++n;
            }
            if (n <= 0) first = -1, n = 0;
          }
          a.dup_groups[3 * tok] = first;
          a.dup_groups[3 * tok + 1] = tok * (K - 1);
          a.dup_groups[3 * tok + 2] = n;
        }
        if (loff < 0) {
          a.dst[slot] = 0;
        } else {
          if (k > 0 && !s.bad) a.dup_loffs[tok * (K - 1) + k - 1] = loff;
          a.dst[slot] = prev >= 0 ? -loff - 1 : loff;
          const int link = (prev >= 0 ? 0 : MOONEP_LINK_PRIMARY) | (next < K ? MOONEP_LINK_HAS_NEXT | s.loff[base + next] : 0);
          meta[c.src_info_off + loff] = slot;
          meta[c.link_off + loff] = link;
          if (a.plan_src_info != nullptr) a.plan_src_info[loff] = slot;
          if (a.plan_link != nullptr) a.plan_link[loff] = link;
        }
      }
      if (in && loff >= 0 && a.weights != nullptr) wbuf[loff] = a.weights[slot];
      if (!a.bulk) {
        copy_plain(c, a, s, t0, ntok, shard);
      } else if (warp < kCopyWarps && ok) {
        ok = copy_bulk(c, a, s, t0, ntok, ring, reinterpret_cast<unsigned char*>(shard));
      }
    }
    if (a.fresh && t_hi == c.S && t_lo < c.S) {
      // token counts above what was routed leave rows that nothing landed in
      __syncthreads();
      for (int e = tid; e < E; e += kThreads)
        for (int g = cur[e]; g < cnt[e] && off[e] + g < NvS; ++g) {
          meta[c.src_info_off + off[e] + g] = -1;
          if (a.plan_src_info != nullptr) a.plan_src_info[off[e] + g] = -1;
          if (a.plan_link != nullptr) a.plan_link[off[e] + g] = 0;
        }
    }
    // all rows of this CTA are in memory before the first of their flags goes out
    bulk_wait<0>();
    fence_gpu();
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    fence_gpu();
    if (ok) {
      visit_pads(c, a, s, cnt, off, zeros, shard, meta, epoch, true);
      for (int i = t_lo * K + tid; i < t_hi * K; i += kThreads) {
        const int d = a.dst[i];
        const int loff = d < 0 ? -d - 1 : d;
        if (loff >= 0 && loff < NvS) st_relaxed_gpu(meta + c.rowflag_off + loff, epoch);
      }
    }
    if (tid == 0) stat_phase(c, MOONEP_PH_BUILD_EXPAND, t_begin);
  }
  // the last CTA publishes what the general kernels' stages publish
  __syncthreads();
  if (tid == 0) {
    fence_gpu();
    if (atomicAdd(c.counters + MOONEP_CTR_DISPATCH_ARRIVE, 1) == (int)gridDim.x - 1) {
      c.counters[MOONEP_CTR_DISPATCH_ARRIVE] = 0;
      fence_sys();
      if (ok && !poisoned(c)) {
        if (a.fresh) {
          const int plan_epoch = abs_epoch(c, MOONEP_FLAG_PLAN, a.epoch_plan);
          st_release_gpu(c.counters + MOONEP_CTR_PLAN_DONE, plan_epoch);
          st_release_sys(flag_ptr(c, 0, MOONEP_FLAG_TPE, 0), abs_epoch(c, MOONEP_FLAG_TPE, a.epoch_tpe));
          st_release_sys(flag_ptr(c, 0, MOONEP_FLAG_PLAN, 0), plan_epoch);
        }
        st_release_sys(flag_ptr(c, 0, MOONEP_FLAG_SENT, 0), abs_epoch(c, MOONEP_FLAG_SENT, a.epoch_sent));
      }
    }
  }
}

// ---- combine ---------------------------------------------------------------------------------------------------

constexpr int kCombineThreads = 512;
constexpr int kCombineRows = 8;  // rows of a token whose loads are in flight together: 128 KB per SM with 32 warps

struct CombineArgs {
  const int* dst;           // [N]
  const uint16_t* in_rows;  // [NvS, H]
  const float* in_w;        // [NvS] or null
  uint16_t* out;            // [S, H]
  float* out_w;             // [S, K] or null
  const int* ready;         // optional: per 128-row block of in_rows, see moonep_combine_push
  int ready_expect;
  int vec_ok;
};

__device__ __forceinline__ void add8(float* acc, const int4& v) {
  acc[0] += bf16lo((unsigned)v.x);
  acc[1] += bf16hi((unsigned)v.x);
  acc[2] += bf16lo((unsigned)v.y);
  acc[3] += bf16hi((unsigned)v.y);
  acc[4] += bf16lo((unsigned)v.z);
  acc[5] += bf16hi((unsigned)v.z);
  acc[6] += bf16lo((unsigned)v.w);
  acc[7] += bf16hi((unsigned)v.w);
}

// A warp per item: 512 bytes of a token's row (vec_ok) or the whole row.  The rows of a token are added in fp32 in
// ascending k and rounded once; a token with one row is copied as it is.
__global__ void __launch_bounds__(kCombineThreads, 2) combine_single_kernel(const MoonepDevCtx c, const CombineArgs a) {
  griddep_wait();
  griddep_launch();
  if (poisoned(c)) return;
  const unsigned long long t_begin = globaltimer_ns();
  const int lane = threadIdx.x & 31;
  const int K = c.K, H = c.H, NvS = c.NvS;
  const int nvec = H / 8;
  const int npieces = a.vec_ok ? (nvec + 31) / 32 : 1;
  const int items = c.S * npieces;  // far below 2^31: S * H elements fit the GPU
  const int step = gridDim.x * (kCombineThreads / 32);
  int it = blockIdx.x * (kCombineThreads / 32) + (threadIdx.x >> 5);
  int d_next = it < items && lane < K ? a.dst[it / npieces * K + lane] : 0;
  for (; it < items; it += step) {
    const int tok = it / npieces, p = it - tok * npieces;
    const int d = d_next;
    if (it + step < items && lane < K) d_next = a.dst[(it + step) / npieces * K + lane];  // not a dependent load then
    int row = d < 0 ? -d - 1 : d;
    const bool valid = lane < K && row >= 0 && row < NvS;
    if (lane < K && !valid) record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_COMBINE_PUSH, 6, d, tok, lane);
    if (!valid) row = -1;
    if (a.ready != nullptr) {
      int got = 1;
      if (valid && ld_acquire_gpu(a.ready + (row >> 7)) - a.ready_expect < 0) {
        const unsigned long long t0 = globaltimer_ns();
        unsigned spins = 0;
        int v;
        while ((v = ld_acquire_gpu(a.ready + (row >> 7))) - a.ready_expect < 0) {
          if ((++spins & 63u) == 0 && (globaltimer_ns() - t0 > c.timeout_ns || poisoned(c))) {
            record_status(c, MOONEP_STATUS_TIMEOUT, MOONEP_K_COMBINE_PUSH, 201, row >> 7, a.ready_expect, v);
            got = 0;
            break;
          }
          __nanosleep(256);
        }
      }
      if (!__all_sync(0xffffffffu, got)) return;
    }
    if (p == 0 && a.in_w != nullptr && a.out_w != nullptr && lane < K)
      a.out_w[(long long)tok * K + lane] = valid ? a.in_w[row] : 0.f;
    const unsigned rows = __ballot_sync(0xffffffffu, valid);
    const bool one = __popc(rows) == 1;
    if (a.vec_ok) {
      const int i = p * 32 + lane;
      float acc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = 0.f;
      int4 only = make_int4(0, 0, 0, 0);
      for (int k0 = 0; k0 < K; k0 += kCombineRows) {
        int4 v[kCombineRows];
#pragma unroll
        for (int r = 0; r < kCombineRows; ++r) {
          const int from = __shfl_sync(0xffffffffu, row, (k0 + r) & 31);
          v[r] = make_int4(0, 0, 0, 0);
          if (k0 + r < K && from >= 0 && i < nvec)
            v[r] = ld16(reinterpret_cast<const int4*>(a.in_rows + (long long)from * H) + i);
        }
#pragma unroll
        for (int r = 0; r < kCombineRows; ++r) {
          if (k0 + r < K && ((rows >> (k0 + r)) & 1u)) {
            add8(acc, v[r]);
            only = v[r];
          }
        }
      }
      if (i < nvec) {
        int4 o = only;
        if (!one) {
          o.x = (int)pack_bf16(acc[0], acc[1]);
          o.y = (int)pack_bf16(acc[2], acc[3]);
          o.z = (int)pack_bf16(acc[4], acc[5]);
          o.w = (int)pack_bf16(acc[6], acc[7]);
        }
        st16(reinterpret_cast<int4*>(a.out + (long long)tok * H) + i, o);
      }
    } else {
      for (int i0 = 0; i0 < H; i0 += 32) {  // whole warps: the shuffles need every lane
        const int i = i0 + lane;
        float acc = 0.f;
        uint16_t only = 0;
        for (int k = 0; k < K; ++k) {
          const int from = __shfl_sync(0xffffffffu, row, k);
          if (from >= 0 && i < H) {
            only = a.in_rows[(long long)from * H + i];
            acc += __uint_as_float((unsigned)only << 16);
          }
        }
        if (i < H) {
          const __nv_bfloat16 b = __float2bfloat16_rn(acc);
          a.out[(long long)tok * H + i] = one ? only : *reinterpret_cast<const uint16_t*>(&b);
        }
      }
    }
  }
  if (threadIdx.x == 0) stat_phase(c, MOONEP_PH_FOLD, t_begin);
}

}  // namespace

}  // namespace moonep

using namespace moonep;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

extern "C" int moonep_single_supported(int E, int S, int K) {
  return E <= kMaxExperts && (long long)S * K <= kMaxEntries ? 1 : 0;
}

extern "C" int moonep_dispatch_single(void* ctx, int fresh, const int* topk, const int* tpe, int* dst, int* cu_seqlens,
                                      int* experts_to_copy, int* zero_fill, int* remote_stats, int* dup_groups,
                                      int* dup_loffs, int* dup_counts, int* plan_src_info, int* plan_link,
                                      const void* hidden, const float* weights, int with_weights, int epoch_tpe,
                                      int epoch_plan, int epoch_sent, int n_ctas, void* stream) {
  auto* h = (HostCtx*)ctx;
  const MoonepDevCtx& c = h->dev;
  if (c.R != 1 || (fresh && !moonep_single_supported(c.E, c.S, c.K))) {
    set_error("moonep_dispatch_single: needs a single rank, at most 4096 experts and 262144 routing entries");
    return 1;
  }
  SingleArgs a;
  a.topk = topk;
  a.tpe = tpe;
  a.dst = dst;
  a.cu_seqlens = cu_seqlens;
  a.experts_to_copy = experts_to_copy;
  a.zero_fill = zero_fill;
  a.remote_stats = remote_stats;
  a.dup_groups = dup_groups;
  a.dup_loffs = dup_loffs;
  a.dup_counts = dup_counts;
  a.plan_src_info = plan_src_info;
  a.plan_link = plan_link;
  a.hidden = (const uint16_t*)hidden;
  a.weights = weights;
  a.with_weights = with_weights;
  a.fresh = fresh;
  a.topk_vec = aligned16(topk) ? 1 : 0;
  a.vec_ok = (c.H % 8 == 0 && aligned16(hidden)) ? 1 : 0;
  a.bulk = a.vec_ok;
  a.epoch_tpe = epoch_tpe;
  a.epoch_plan = epoch_plan;
  a.epoch_sent = epoch_sent;
  const size_t static_bytes = sizeof(SingleShared) + 1024;
  const size_t limit = (size_t)imax(0, h->max_smem_optin - (int)static_bytes);
  const size_t tables = fresh ? (size_t)3 * c.E * sizeof(int) : 0;
  a.piece_bytes = 0;
  a.npieces = 1;
  if (a.bulk) {
    const long long row_bytes = (long long)c.H * 2;
    const long long room = (long long)(limit - tables) / (kCopyWarps * kRing + 1) / 16 * 16;
    const long long most = room < kMaxPiece ? room : kMaxPiece;
    a.npieces = (int)((row_bytes + most - 1) / most);
    a.piece_bytes = (int)(((row_bytes + a.npieces - 1) / a.npieces + 15) / 16 * 16);
  }
  const size_t smem = (size_t)(kCopyWarps * kRing + 1) * a.piece_bytes + tables;
  if (int rc = check_cuda(cudaFuncSetAttribute(dispatch_single_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit),
                          "cudaFuncSetAttribute(dispatch_single_kernel)"))
    return rc;
  int grid = imax(1, imin(c.local_sms, h->sm_count));
  if (n_ctas > 0) grid = imin(grid, n_ctas);
  a.tokens_per_cta = (c.S + grid - 1) / grid;
  if (int rc = check_cuda(launch_maybe_pdl(dispatch_single_kernel, grid, kThreads, smem, (cudaStream_t)stream,
                                           h->enable_pdl != 0, c, a),
                          "launch dispatch_single_kernel"))
    return rc;
  return check_launch("dispatch_single_kernel");
}

extern "C" int moonep_combine_single(void* ctx, const int* dst, const void* in_rows, const float* in_w, void* out,
                                     float* out_w, const int* ready, int ready_expect, void* stream) {
  auto* h = (HostCtx*)ctx;
  const MoonepDevCtx& c = h->dev;
  if (c.R != 1) {
    set_error("moonep_combine_single: needs a single rank");
    return 1;
  }
  CombineArgs a;
  a.dst = dst;
  a.in_rows = (const uint16_t*)in_rows;
  a.in_w = in_w;
  a.out = (uint16_t*)out;
  a.out_w = out_w;
  a.ready = ready;
  a.ready_expect = ready_expect;
  a.vec_ok = (c.H % 8 == 0 && aligned16(in_rows) && aligned16(out)) ? 1 : 0;
  const long long items = (long long)c.S * (a.vec_ok ? (c.H / 8 + 31) / 32 : 1);
  const long long need = (items + kCombineThreads / 32 - 1) / (kCombineThreads / 32);
  const int most = 2 * imax(1, imin(c.local_sms, h->sm_count));
  const int grid = need < most ? (int)need : most;
  if (int rc = check_cuda(launch_maybe_pdl(combine_single_kernel, grid, kCombineThreads, 0, (cudaStream_t)stream,
                                           h->enable_pdl != 0, c, a),
                          "launch combine_single_kernel"))
    return rc;
  return check_launch("combine_single_kernel");
}
