// Dispatch and combine of a Buffer with one rank, for sm_100a.
//
// With one rank nothing crosses a link and nothing is balanced: every routing entry lands on this GPU, the group
// layout is a prefix sum over the padded token counts, and the K entries of a token are one duplicate group.  The
// general kernels (dispatch.cu, combine_push.cu) reach that result through a chain of grid-wide hand-offs (publish,
// table stage on one CTA, token stage, link words walked by the expand role) which took 45 us of the 205 us of a
// dispatch at S=4096, H=7168, K=8, E=256 before most rows were written, and 65 of 84 us at S=16.  Here
//
//   dispatch   one launch whose CTAs wait for nobody.  Every CTA derives the whole group layout itself (E counts, one
//              prefix sum).  Four warps clear pad rows with bulk stores from a piece of zeros, handed out from one
//              counter; the others count the routing entries before the CTA's own contiguous range of tokens, give its
//              entries their rows and publish "planned"; then up to six of them stream tokens through shared memory,
//              one bulk load and K bulk stores per row.  A CTA that is done with its tokens takes rows over from CTAs that
//              have planned theirs: SMs reach HBM at rates that differ by a quarter, and with a fixed share per SM the
//              kernel took 138 (426) us at S=4096 (16384) where its average CTA was done after 117 (363); now 131 (400).
//   combine    a warp per 512-byte piece of an output row (several at once where a token has few rows), straight from the
//              token's K destinations: no work counter, no lists.
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
constexpr int kRing = 3;           // stages per ring: two loads run ahead of the stores
constexpr int kMaxStage = 16384;   // bytes
constexpr int kZeroBytes = 8192;
constexpr int kPlanWarps = 12;     // warps 0..11 plan, then up to kCopyWarps of them copy; warps 12..15 clear pad rows
// 4 with 14 KB rows, whose rings fill shared memory.  With more than 6 warps the stores an SM has queued outweigh what
// they hide: 12 warps took 28 us where 6 take 22 at S=1777, H=2056, K=5; 3 warps took 102 us where 6 take 97 at S=8192,
// H=4096, K=6.
constexpr int kCopyWarps = 6;
constexpr int kEntries = kPlanWarps * 32;  // routing entries planned at a time (whole tokens)
// A copy warp asks for its tokens one at a time, and in the end looks through the other CTAs' counters for what is left: about
// 4 us of latency, for which a CTA with little to move waits longer than for the slowest SM.  So up to kDealtBytes read and
// written per CTA the tokens are dealt to its warps at once.  Dispatch of S=2048, H=2048, K=4 24.1 -> 20.5 us, S=1024, H=4096,
// K=2 21.5 -> 18.0, S=4096, H=1024, K=8 30.2 -> 28.2; with 1 MB per CTA (S=2048, H=4096, K=8) it would be 50.5 -> 52.2.
constexpr long long kDealtBytes = 768 << 10;
constexpr int kDealtRounds = 6;
// Rows that share a stage at most, as far as the rings of six warps have room and the CTA's tokens make equal shares for them.  A
// unit costs a copy warp a chain of round trips, and an SM has more on its way with more in a stage.  Against rows that fill
// 4 KB, dispatch and combine, us: S=16384, K=4, H=1000 79.3 -> 74.9, H=2048 135.2 -> 127.9; S=4096, K=8, H=2048 64.2 -> 61.4.
// Stages of 16 KB for four warps make the dispatch alone another 2 to 5 % shorter, but the combine behind it longer by more
// (S=16384, K=4: H=2048 132.9 together, H=4096 249.6 instead of 237.7).  Equal shares lose where they are smaller than a stage's
// worth: a replay of S=4096, H=256, K=8 (units of five rows, not eight) takes 16.3 us where it took 15.9, S=2048 14.8 (15.8), S=8192
// 22.8 (24.9).
constexpr int kUnitTokens = 8;
constexpr int kUnits = 64;         // units remembered per copy warp: those loaded and those not flagged yet
constexpr int kGrabs = 64;         // grabs of pad rows remembered per warp
constexpr int kMaxGroups = 4096;   // experts, and prefetch slots: up to four words of shared memory each
// Every CTA reads the routing before its own tokens, beside the copies of the CTAs that are ahead.  The line is how far the
// kernel is tested, not where the general kernels catch up: S=32768, K=8, H=1024 (at the line) takes 165 us here and 363
// there, and with the line out of the way S=65536 takes 302 and 725, S=262144, H=64 498 and 2816.
constexpr int kMaxEntries = 1 << 18;
// work[]: pad rows handed out, then per CTA the tokens handed out, then per CTA the epoch at which its tokens were planned
constexpr int kMaxCtas = 256;
constexpr int kWorkPads = 0, kWorkNext = 1, kWorkReady = kWorkNext + kMaxCtas;

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
  // [NvS, H] or null: a copy of the shard, made on the way by a second store of every piece instead of a pass that reads
  // the shard again (S=8192, H=4096, K=6, E=64: 364 -> 293 us per round trip).  Fresh plans only: a replay does not know
  // which rows no group uses.
  uint16_t* out;
  float* out_w;   // [NvS] or null: of its weights
  const uint16_t* hidden;  // [S, H]
  const float* weights;    // [S, K] or null
  int with_weights;        // pad rows' weight slots are cleared
  int fresh;
  int exact;     // fresh: counts that do not add up to the routing entries are an index error, not rows left unused
  int topk_vec;  // topk can be read 16 bytes at a time
  int vec_ok;    // rows of the shard and the copy are whole 16-byte words at 16-byte addresses
  int bulk_pads; // pads are cleared in bulk stores
  int bulk;      // rows go through shared memory with bulk copies
  int word;      // bytes per store of a row that does not
  int narrow;    // its input is read two bytes at a time
  int stage_bytes, npieces;  // a row is moved in npieces pieces of at most stage_bytes
  int copy_warps;            // warps that stream rows, each through a ring of its own
  int tokens_per_unit;       // whole rows that share a stage (npieces == 1)
  int rounds;                // units of its CTA that a copy warp gets without asking
  int pads_per_grab;         // at least
  int tokens_per_cta;
  uint16_t* shard;
  int* meta;
  int* work;
  int epoch_tpe, epoch_plan, epoch_sent;
};

// What a copy warp moves at a time: rows [tok, tok + ntok) of the input, or bytes [off, off + len) of one row.
struct Unit {
  int tok, ntok;
  unsigned off, len;
};

struct SingleShared {
  unsigned long long bar[kCopyWarps * kRing];
  Unit unit[kCopyWarps][kUnits];
  int2 warp_sum[kWarps];
  int grab[kWarps - kPlanWarps][kGrabs];
  int loff[kEntries];  // destination row of every entry in hand, -1: none
  int bad;             // entries in hand without a row
  int last;
};

__device__ __forceinline__ void plan_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kPlanWarps * 32) : "memory"); }

// Inclusive prefix sums of two values over the threads of the CTA; all threads call it.
__device__ __forceinline__ int2 block_scan(int2 v, int2* warp_sum, int2& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, v.x, o), y = __shfl_up_sync(0xffffffffu, v.y, o);
    if (lane >= o) v.x += x, v.y += y;
  }
  if (lane == 31) warp_sum[warp] = v;
  __syncthreads();
  int2 before = make_int2(0, 0);
  total = make_int2(0, 0);
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int2 x = warp_sum[w];
    if (w < warp) before.x += x.x, before.y += x.y;
    total.x += x.x, total.y += x.y;
  }
  __syncthreads();
  return make_int2(v.x + before.x, v.y + before.y);
}

__device__ __forceinline__ int padded_rows(int cnt, int P) { return cnt > 0 ? ((cnt + P - 1) / P) * P : 0; }

// Group layout in shared memory: cnt/off of every expert (fresh plans) and the running total of pad rows per group.
struct Layout {
  const int* first;  // replay: first pad row of a group
  const int* cnt;    // fresh
  const int* off;    // fresh
  const int* cum;    // inclusive running total of pad rows
  int groups;
  __device__ int pad_row(int j) const {
    int lo = 0, hi = groups - 1;  // first group whose running total exceeds j
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (cum[mid] > j) hi = mid; else lo = mid + 1;
    }
    const int start = cnt != nullptr ? off[lo] + cnt[lo] : first[lo];
    return start + (j - (lo > 0 ? cum[lo - 1] : 0));
  }
};

// A warp clears n elements at any address: 16-byte stores between the edges.
__device__ __forceinline__ void clear_row(uint16_t* p, int n) {
  const int lane = threadIdx.x & 31;
  const int head = min(n, (int)((16u - ((unsigned)reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) / 2);
  const int words = (n - head) / 8, tail = head + words * 8;
  if (lane < head) p[lane] = 0;
  for (int i = lane; i < words; i += 32) st16(reinterpret_cast<int4*>(p + head) + i, make_int4(0, 0, 0, 0));
  if (lane < n - tail) p[tail + lane] = 0;
}

// Warps kPlanWarps.. : clear pad rows (and their weights), mark them unused in a fresh plan.  Rows are handed out from
// one counter, some at a time, a lane per row.  Their row flags are released at the end, behind one wait and one
// fence: a fence per grab held the clears of S=128, H=7168, E=256 (31 K pad rows) to 5.3 TB/s.
__device__ void clear_pads(const MoonepDevCtx& c, const SingleArgs& a, const Layout& lay, int* grabs,
                           const unsigned char* zeros, uint16_t* shard, int* meta, int epoch) {
  const int lane = threadIdx.x & 31;
  const long long row_bytes = (long long)c.H * 2;
  const int total = lay.groups > 0 ? lay.cum[lay.groups - 1] : 0;
  // a sixth of a warp's share at a time where there are many: the grabs of 592 warps meet at one address (two rows per
  // grab: 100 us per round trip at S=128, H=7168, E=256 with 31 K pad rows; eight: 91)
  const int per = max(a.pads_per_grab, min(32, total / ((int)gridDim.x * (kWarps - kPlanWarps) * 6)));
  auto row_of = [&](int j) {
    const int row = lane < per && j + lane < total ? lay.pad_row(j + lane) : -1;
    return row < c.NvS ? row : -1;
  };
  int held = 0;
  auto flag_all = [&]() {
    bulk_wait<0>();
    fence_gpu();
    __syncwarp();
    for (int q = 0; q < held; ++q) {
      const int row = row_of(grabs[q]);
      if (row >= 0) st_relaxed_gpu(meta + c.rowflag_off + row, epoch);
    }
    held = 0;
    __syncwarp();
  };
  for (;;) {
    int j = 0;
    if (lane == 0) j = atomicAdd(a.work + kWorkPads, per);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= total) break;
    const int row = row_of(j);
    if (row >= 0) {
      if (a.bulk_pads) {
        unsigned char* p = reinterpret_cast<unsigned char*>(shard) + row * row_bytes;
        unsigned char* p2 = reinterpret_cast<unsigned char*>(a.out) + row * row_bytes;
        for (long long o = 0; o < row_bytes; o += kZeroBytes) {
          const unsigned len = (unsigned)min((long long)kZeroBytes, row_bytes - o);
          bulk_s2g(p + o, zeros, len);
          if (a.out != nullptr) bulk_s2g(p2 + o, zeros, len);
        }
      }
      if (a.with_weights) reinterpret_cast<float*>(meta + c.weights_off)[row] = 0.f;
      if (a.out_w != nullptr) a.out_w[row] = 0.f;
      if (a.fresh) {
        meta[c.src_info_off + row] = -1;
        if (a.plan_src_info != nullptr) a.plan_src_info[row] = -1;
        if (a.plan_link != nullptr) a.plan_link[row] = 0;
      }
    }
    bulk_commit();
    bulk_wait_read<3>();  // what an SM has queued stays small, so that the rows go to the SMs that are fastest
    if (!a.bulk_pads) {
      for (int q = 0; q < per; ++q) {
        const int r = __shfl_sync(0xffffffffu, row, q);
        if (r < 0) continue;
        clear_row(shard + (long long)r * c.H, c.H);
        if (a.out != nullptr) clear_row(a.out + (long long)r * c.H, c.H);
      }
      fence_gpu();  // other lanes' stores precede the flag that lane q releases
    }
    if (lane == 0) grabs[held] = j;
    __syncwarp();
    if (++held == kGrabs) flag_all();
  }
  flag_all();
}

// Hands out units to a copy warp: those of its own CTA, then, from CTAs whose tokens are planned, whatever is left.
struct Units {
  const MoonepDevCtx& c;
  const SingleArgs& a;
  const int epoch;
  int tok, piece;  // a row moved in several pieces: the piece that comes next
  int state;  // 0: the units that are this warp's from the start, 1: more of the own CTA's, 2: other CTAs'
  int round;

  __device__ int count_of(int cta) const { return max(0, min(c.S - cta * a.tokens_per_cta, a.tokens_per_cta)); }
  // tokens of a CTA that are dealt to its warps without the counter
  __device__ int dealt() const { return a.rounds * a.copy_warps * a.tokens_per_unit; }

  __device__ bool take(int cta, Unit& u) {
    int g = 0;
    if ((threadIdx.x & 31) == 0) g = dealt() + atomicAdd(a.work + kWorkNext + cta, a.tokens_per_unit);
    return unit_at(cta, __shfl_sync(0xffffffffu, g, 0), u);
  }

  __device__ bool unit_at(int cta, int g, Unit& u) {
    const int n = count_of(cta);
    if (g >= n) return false;
    const long long row_bytes = (long long)c.H * 2;
    u.tok = cta * a.tokens_per_cta + g;
    u.ntok = min(a.tokens_per_unit, n - g);
    u.off = 0;
    u.len = a.npieces > 1 ? a.stage_bytes : (unsigned)(u.ntok * row_bytes);
    tok = u.tok;
    piece = 1;
    return true;
  }

  // The units that need no counter: the next piece of a row, and those that are this warp's from the start.
  __device__ bool next_dealt(Unit& u) {
    if (piece < a.npieces) {
      u.tok = tok;
      u.ntok = 1;
      u.off = (unsigned)(piece * a.stage_bytes);
      u.len = min((unsigned)a.stage_bytes, (unsigned)(c.H * 2) - u.off);
      ++piece;
      return true;
    }
    if (state == 0 && round < a.rounds) {
      const int g = (round++ * a.copy_warps + (int)(threadIdx.x >> 5)) * a.tokens_per_unit;
      if (unit_at(blockIdx.x, g, u)) return true;
    }
    if (state == 0) state = 1;
    return false;
  }

  __device__ bool next(Unit& u) {
    const int lane = threadIdx.x & 31;
    if (next_dealt(u)) return true;
    if (a.tokens_per_cta <= dealt()) return false;  // nothing beyond what was dealt, here or elsewhere
    if (state == 1) {
      if (take(blockIdx.x, u)) return true;
      state = 2;
    }
    for (;;) {
      int left[kMaxCtas / 32], ready[kMaxCtas / 32];
#pragma unroll
      for (int i = 0; i < kMaxCtas / 32; ++i) {  // independent loads, all in flight together
        const int v = i * 32 + lane;
        left[i] = 0;
        ready[i] = epoch;
        if (v < (int)gridDim.x) {
          left[i] = count_of(v) - dealt() - ld_volatile(a.work + kWorkNext + v);
          if (a.fresh) ready[i] = ld_volatile(a.work + kWorkReady + v);
        }
      }
      int most = 0, victim = -1;  // the CTA with the most tokens left; among equals another one for every thief
#pragma unroll
      for (int i = 0; i < kMaxCtas / 32; ++i)
        if (left[i] > most && ready[i] - epoch >= 0) {
          most = left[i];
          victim = i * 32 + lane;
        }
      const int best = __reduce_max_sync(0xffffffffu, most);
      if (best <= 0) return false;
      const unsigned cand = __ballot_sync(0xffffffffu, most == best);
      const unsigned after = cand & ~((2u << (blockIdx.x & 31)) - 1u);
      victim = __shfl_sync(0xffffffffu, victim, __ffs(after ? after : cand) - 1);
      if (a.fresh) ld_acquire_gpu(a.work + kWorkReady + victim);  // what it planned is visible from here on
      if (take(victim, u)) return true;
    }
  }
};

// A copy warp: units go global -> shared -> their K destination rows; a lane per (row, destination) issues the store.
// Row flags are released at the end, or when the list of units is full, behind one wait and one fence.  The units that are the
// warp's from the start are asked for before their tokens are planned (start).
struct CopyWarp {
  const MoonepDevCtx& c;
  const SingleArgs& a;
  SingleShared& s;
  unsigned char* ring;
  Units from;
  int loaded, more;

  __device__ CopyWarp(const MoonepDevCtx& c_, const SingleArgs& a_, SingleShared& s_, unsigned char* stages, int epoch)
      : c(c_), a(a_), s(s_), ring(stages + (size_t)(threadIdx.x >> 5) * kRing * a_.stage_bytes),
        from{c_, a_, epoch, 0, a_.npieces, 0, 0}, loaded(0), more(1) {}

  __device__ void issue(const Unit& u) {
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
      s.unit[warp][loaded % kUnits] = u;
      const int q = loaded % kRing;
      unsigned long long* bar = s.bar + warp * kRing + q;
      mbar_expect_tx(bar, u.len);
      bulk_g2s(ring + (size_t)q * a.stage_bytes,
               reinterpret_cast<const unsigned char*>(a.hidden) + u.tok * (c.H * 2ll) + u.off, u.len, bar);
    }
    __syncwarp();
    ++loaded;
  }

  __device__ void start() {
    Unit u;
    while (loaded < kRing - 1 && from.next_dealt(u)) issue(u);
  }

  __device__ bool load() {
    Unit u;
    if (!from.next(u)) return false;
    issue(u);
    return true;
  }

  __device__ bool run(unsigned char* shard, int* meta, int epoch, int t_lo, int t_hi);
};

// [t_lo, t_hi): tokens whose rows are listed in s.loff.
__device__ bool CopyWarp::run(unsigned char* shard, int* meta, int epoch, int t_lo, int t_hi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row_bytes = (long long)c.H * 2;
  const int K = c.K, NvS = c.NvS;
  unsigned long long* bar = s.bar + warp * kRing;
  const Unit* units = s.unit[warp];
  int stored = 0;
  auto row_of = [&](const Unit& u, int e) {
    if (u.tok >= t_lo && u.tok < t_hi) return s.loff[(u.tok - t_lo) * K + e];
    const int d = a.dst[u.tok * K + e];
    const int loff = d < 0 ? -d - 1 : d;
    return loff >= 0 && loff < NvS ? loff : -1;
  };
  int flagged = 0;
  auto flag_stored = [&]() {  // a lane flags the rows it has stored itself
    bulk_wait<0>();
    fence_gpu();
    for (; flagged < stored; ++flagged) {
      const Unit u = units[flagged % kUnits];
      if (u.ntok == 1 && u.off + u.len < row_bytes) continue;  // more pieces of the row follow
      for (int e = lane; e < u.ntok * K; e += 32) {
        const int loff = row_of(u, e);
        if (loff >= 0) st_relaxed_gpu(meta + c.rowflag_off + loff, epoch);
      }
    }
    __syncwarp();
  };
  while (loaded < kRing - 1 && more) more = load();
  while (stored < loaded) {
    const Unit u = units[stored % kUnits];
    const int q = stored % kRing;
    const int mine = lane < u.ntok * K ? row_of(u, lane) : -1;
    const bool got = mbar_wait(bar + q, (unsigned)((stored / kRing) & 1), c.timeout_ns);
    if (!__all_sync(0xffffffffu, got)) {
      if (lane == 0) record_status(c, MOONEP_STATUS_TIMEOUT, MOONEP_K_DISPATCH_EXPAND, 100, q, stored, u.tok);
      for (int n = stored; n < loaded; ++n)  // nothing may land in shared memory after the CTA has left
        mbar_wait(bar + n % kRing, (unsigned)((n / kRing) & 1), c.timeout_ns);
      return false;
    }
    const unsigned len = u.ntok > 1 ? (unsigned)row_bytes : u.len;
    for (int e = lane; e < u.ntok * K; e += 32) {
      const int loff = e < 32 ? mine : row_of(u, e);
      if (loff < 0) continue;
      const unsigned char* src = ring + (size_t)q * a.stage_bytes + (e / K) * row_bytes;
      bulk_s2g(shard + loff * row_bytes + u.off, src, len);
      if (a.out != nullptr) bulk_s2g(reinterpret_cast<unsigned char*>(a.out) + loff * row_bytes + u.off, src, len);
    }
    bulk_commit();
    ++stored;
    if (more) {
      bulk_wait_read<1>();  // the stage to refill was stored from one unit ago
      __syncwarp();
      more = load();
    }
    if (loaded - flagged == kUnits) flag_stored();
  }
  flag_stored();
  return true;
}

// The same without bulk copies: words of D for this CTA's tokens, loaded as they are or (input rows that start anywhere)
// two bytes at a time.  A warp takes kPlainWords words per lane at a time, so that one token keeps several warps busy and a
// lane several loads in flight.  Against a warp per row that moved (and cleared) two bytes per lane: S=4096, K=8, H=4096 with
// an input that is not 16-byte aligned 1059 -> 84 us, S=128, H=7168 609 -> 33, S=4096, K=4, H=4100 665 -> 86.
constexpr int kPlainWords = 4;

template <typename D, typename T>
__device__ void copy_words(const MoonepDevCtx& c, const SingleArgs& a, int t_lo, int t_hi, uint16_t* shard) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = c.H * 2 / (int)sizeof(D), pieces = (n + 32 * kPlainWords - 1) / (32 * kPlainWords);
  for (int u = warp; u < (t_hi - t_lo) * pieces; u += kPlanWarps) {
    const int tok = t_lo + u / pieces, i0 = (u % pieces) * 32 * kPlainWords + lane;
    const T* src = reinterpret_cast<const T*>(a.hidden + (long long)tok * c.H);
    const int d = lane < c.K ? a.dst[tok * c.K + lane] : 0;
    int loff = d < 0 ? -d - 1 : d;
    if (lane >= c.K || loff < 0 || loff >= c.NvS) loff = -1;
    D v[kPlainWords];
#pragma unroll
    for (int q = 0; q < kPlainWords; ++q) {
      T* part = reinterpret_cast<T*>(v + q);
#pragma unroll
      for (int p = 0; p < (int)(sizeof(D) / sizeof(T)); ++p)
        if (i0 + q * 32 < n) part[p] = src[(long long)(i0 + q * 32) * (sizeof(D) / sizeof(T)) + p];
    }
    for (int k = 0; k < c.K; ++k) {
      const int row = __shfl_sync(0xffffffffu, loff, k);
      if (row < 0) continue;
      for (uint16_t* base : {shard, a.out}) {
        if (base == nullptr) continue;
        D* to = reinterpret_cast<D*>(base + (long long)row * c.H) + i0;
#pragma unroll
        for (int q = 0; q < kPlainWords; ++q)
          if (i0 + q * 32 < n) to[q * 32] = v[q];
      }
    }
  }
}

__device__ void copy_plain(const MoonepDevCtx& c, const SingleArgs& a, int t_lo, int t_hi, uint16_t* shard, int* meta,
                           int epoch) {
  switch (a.word) {
    case 16:
      if (a.narrow) copy_words<int4, uint16_t>(c, a, t_lo, t_hi, shard); else copy_words<int4, int4>(c, a, t_lo, t_hi, shard);
      break;
    case 8: copy_words<int2, int2>(c, a, t_lo, t_hi, shard); break;
    case 4: copy_words<int, int>(c, a, t_lo, t_hi, shard); break;
    default: copy_words<uint16_t, uint16_t>(c, a, t_lo, t_hi, shard);
  }
  fence_gpu();
  plan_sync();  // a row's words come from several warps
  fence_gpu();
  for (int e = t_lo * c.K + threadIdx.x; e < t_hi * c.K; e += kEntries) {
    const int d = a.dst[e];
    const int loff = d < 0 ? -d - 1 : d;
    if (loff >= 0 && loff < c.NvS) st_relaxed_gpu(meta + c.rowflag_off + loff, epoch);
  }
}

// Rows [lo, hi) of the shard, which the dispatch does not write, as they are into the copy; thread `t` of `n`.
__device__ void copy_tail(const MoonepDevCtx& c, const SingleArgs& a, const int* meta, int lo, int hi, int t, int n) {
  const uint16_t* shard = c.hidden_peer[0];
  const long long e0 = (long long)lo * c.H, e1 = (long long)hi * c.H;
  if (a.vec_ok) {
    const int4* src = reinterpret_cast<const int4*>(shard);
    int4* dst = reinterpret_cast<int4*>(a.out);
    for (long long i = e0 / 8 + t; i < e1 / 8; i += 4ll * n) {
      int4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + (long long)u * n < e1 / 8) v[u] = ld16(src + i + (long long)u * n);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + (long long)u * n < e1 / 8) st16(dst + i + (long long)u * n, v[u]);
    }
  } else {
    for (long long i = e0 + t; i < e1; i += n) a.out[i] = shard[i];
  }
  if (a.out_w != nullptr)
    for (int i = lo + t; i < hi; i += n) a.out_w[i] = reinterpret_cast<const float*>(meta + c.weights_off)[i];
}

// What a thread of the planning warps asks for before the group layout is known: the entries before the CTA's tokens that it
// counts first, and the first entry that it plans, with its weight.  Beside other CTAs' rows and pads each of these round trips
// takes microseconds.  With them, and the first rows of the copy warps, asked for where they were used: last CTA planned 21 us
// after the layout where it takes 12 (S=4096, K=8, E=256) and 4.5 (3.5; S=2048, K=4, E=16), kernel 39.5 (37.5; S=2048, H=4096,
// K=8) and 15.0 (12.4; S=2048, H=2048, K=4).  Among many large pad rows (H=8192, K=8, E=64) neither kernel is slower by itself, but
// the round trips of two sizes are: S=200 41.8 -> 41.3, S=300 44.4 -> 45.2, S=450 48.8 -> 49.9, S=600 51.2 -> 49.8.  Counting in
// bytes per thread instead of atomics gained nothing beyond that.
constexpr int kCountLoads = 8;
struct Early {
  int4 v[kCountLoads];
  int e;
  float w;
};

__device__ __forceinline__ Early load_early(const SingleArgs& a, int K, int before, int t_lo, int t_hi) {
  Early p;
  const int tid = threadIdx.x, nv = a.topk_vec ? before / 4 : 0;
  const bool mine = tid < kEntries / K * K && t_lo * K + tid < t_hi * K;
  p.e = mine ? a.topk[t_lo * K + tid] : -1;
  p.w = mine && a.weights != nullptr ? a.weights[t_lo * K + tid] : 0.f;
#pragma unroll
  for (int u = 0; u < kCountLoads; ++u)
    p.v[u] = tid + u * kEntries < nv ? __ldg(reinterpret_cast<const int4*>(a.topk) + tid + u * kEntries) : make_int4(-1, -1, -1, -1);
  return p;
}

// Threads of the planning warps: rows for the entries of tokens [t_lo, t_hi), and everything the plan says about them.
__device__ void plan_tokens(const MoonepDevCtx& c, const SingleArgs& a, SingleShared& s, const Early& early, const int* cnt,
                            const int* off, int* cur, int* meta, int before, int t_lo, int t_hi) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int E = c.E, K = c.K, NvS = c.NvS;
  float* wbuf = reinterpret_cast<float*>(meta + c.weights_off);
  // routing entries before this CTA's tokens
  const int nv = a.topk_vec ? before / 4 : 0;
  auto count = [&](int e) {
    if ((unsigned)e < (unsigned)E) atomicAdd(cur + e, 1);
  };
  // half of a thread's loads are on their way while it counts the other half
  int4 v[kCountLoads];
#pragma unroll
  for (int u = 0; u < kCountLoads; ++u) v[u] = early.v[u];
  for (int i0 = tid; i0 < nv; i0 += kCountLoads * kEntries) {
#pragma unroll
    for (int u0 = 0; u0 < kCountLoads; u0 += kCountLoads / 2) {
#pragma unroll
      for (int u = u0; u < u0 + kCountLoads / 2; ++u) {
        count(v[u].x);
        count(v[u].y);
        count(v[u].z);
        count(v[u].w);
        const int i = i0 + (kCountLoads + u) * kEntries;
        v[u] = i < nv ? __ldg(reinterpret_cast<const int4*>(a.topk) + i) : make_int4(-1, -1, -1, -1);
      }
    }
  }
  for (int i = nv * 4 + tid; i < before; i += kEntries) count(a.topk[i]);
  const int tokens_per_step = kEntries / K;
  for (int t0 = t_lo; t0 < t_hi; t0 += tokens_per_step) {
    const int nent = min(tokens_per_step, t_hi - t0) * K, slot = t0 * K + tid;
    const bool in = tid < nent;
    int e = !in ? -1 : t0 == t_lo ? early.e : a.topk[slot];
    const float weight = t0 == t_lo ? early.w : in && a.weights != nullptr ? a.weights[slot] : 0.f;
    if (in && (unsigned)e >= (unsigned)E) {
      record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_PLAN_TOKENS, 2, e, E, slot);
      e = -1;
    }
    plan_sync();  // the entries before are counted; the step before is done with s.loff and s.bad
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
      plan_sync();
    }
    int loff = -1;
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
    if (in) {
      s.loff[tid] = loff;
      if (loff < 0) s.bad = 1;
    }
    plan_sync();
    if (!in) continue;
    // all entries of a token land on this rank: the first is its primary row, the others its duplicates in order
    const int k = tid % K, base = tid - k, tok = slot / K;
    int prev = k - 1, next = k + 1;
    if (s.bad) {  // some entry has no row (recorded above): skip such entries
      while (prev >= 0 && s.loff[base + prev] < 0) --prev;
      while (next < K && s.loff[base + next] < 0) ++next;
    }
    if (K > 1 && k == 0) {
      int first = loff, n = K - 1;
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
      continue;
    }
    if (k > 0 && !s.bad) a.dup_loffs[tok * (K - 1) + k - 1] = loff;
    a.dst[slot] = prev >= 0 ? -loff - 1 : loff;
    const int link = (prev >= 0 ? 0 : MOONEP_LINK_PRIMARY) | (next < K ? MOONEP_LINK_HAS_NEXT | s.loff[base + next] : 0);
    meta[c.src_info_off + loff] = slot;
    meta[c.link_off + loff] = link;
    if (a.plan_src_info != nullptr) a.plan_src_info[loff] = slot;
    if (a.plan_link != nullptr) a.plan_link[loff] = link;
    if (a.weights != nullptr) {
      wbuf[loff] = weight;
      if (a.out_w != nullptr) a.out_w[loff] = weight;
    }
  }
  if (t_hi == c.S) {
    // token counts above what was routed leave rows that nothing landed in
    plan_sync();
    for (int e = tid; e < E; e += kEntries)
      for (int g = cur[e]; g < cnt[e]; ++g) {
        const int row = off[e] + g;
        if (row < 0 || row >= NvS) break;  // absurd counts: recorded by CTA 0
        meta[c.src_info_off + row] = -1;
        if (a.plan_src_info != nullptr) a.plan_src_info[row] = -1;
        if (a.plan_link != nullptr) a.plan_link[row] = 0;
        if (a.out != nullptr) copy_tail(c, a, meta, row, row + 1, 0, 1);
      }
  }
}

__global__ void __launch_bounds__(kThreads, 1) dispatch_single_kernel(const MoonepDevCtx c, const SingleArgs a) {
  extern __shared__ __align__(128) unsigned char s_dyn[];  // rings, zeros, the group layout
  __shared__ __align__(8) SingleShared s;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int E = c.E, K = c.K, NvS = c.NvS;
  unsigned char* zeros = s_dyn + (size_t)a.copy_warps * kRing * a.stage_bytes;
  int* tables = reinterpret_cast<int*>(zeros + (a.bulk_pads ? kZeroBytes : 0));
  if (tid < kCopyWarps * kRing) mbar_init(s.bar + tid, 1);
  if (a.bulk_pads)
    for (int i = tid; i < kZeroBytes / 16; i += kThreads) reinterpret_cast<int4*>(zeros)[i] = make_int4(0, 0, 0, 0);
  fence_barrier_init();
  fence_proxy_async();
  griddep_wait();
  griddep_launch();
  const unsigned long long t_begin = globaltimer_ns();
  // what the kernel begins with, in one round trip to memory
  const int epoch = abs_epoch(c, MOONEP_FLAG_SENT, a.epoch_sent);
  const int first_count = a.fresh && tid < E ? a.tpe[tid] : 0;
  const int t_lo = min(c.S, (int)blockIdx.x * a.tokens_per_cta), t_hi = min(c.S, t_lo + a.tokens_per_cta);
  const int before = t_lo * K;  // routing entries before this CTA's tokens
  Early early;
  if (a.fresh && warp < kPlanWarps) early = load_early(a, K, before, t_lo, t_hi);
  // one answer for the CTA: the code below contains barriers
  const bool run = __syncthreads_and(poisoned(c) ? 0 : 1) != 0;
  bool ok = run;
  if (run) {
    int* meta = a.meta;
    uint16_t* shard = a.shard;
    CopyWarp copier(c, a, s, s_dyn, epoch);
    if (a.bulk && warp < a.copy_warps && t_lo < t_hi) copier.start();
    Layout lay = {nullptr, nullptr, nullptr, nullptr, 0};
    int *cnt = tables, *off = tables + E, *cur = tables + 2 * E;
    int used = NvS;
    if (a.fresh) {
      int* cum = tables + 3 * E;
      int carry = 0, pads = 0;
      for (int e0 = 0; e0 < E; e0 += kThreads) {
        const int e = e0 + tid;
        const int n = e0 == 0 ? first_count : e < E ? a.tpe[e] : 0;
        const int rows = padded_rows(n, c.token_padding);
        int2 total;
        const int2 sum = block_scan(make_int2(rows, rows > 0 ? rows - n : 0), s.warp_sum, total);
        if (e < E) {
          cnt[e] = n;
          off[e] = carry + sum.x - rows;
          cur[e] = 0;
          cum[e] = pads + sum.y;
        }
        carry += total.x;
        pads += total.y;
      }
      used = min(max(carry, 0), NvS);
      lay = {nullptr, cnt, off, cum, E};
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
        for (int b = tid; b < c.B; b += kThreads) {  // a single rank has no use for its prefetch slots
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
        if (tid == 0 && a.exact && carry - pads != c.S * K)
          record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_PLAN_TABLES, 5, carry - pads, c.S * K, 0);
        __syncthreads();
        if (tid == 0) {
          __threadfence();
          st_release_gpu(c.counters + MOONEP_CTR_TABLES_READY, abs_epoch(c, MOONEP_FLAG_PLAN, a.epoch_plan));
        }
      }
    } else if (a.zero_fill != nullptr) {
      const int groups = E + c.B;
      int *first = tables, *cum = tables + groups;
      int pads = 0;
      for (int g0 = 0; g0 < groups; g0 += kThreads) {
        const int g = g0 + tid;
        const int2 range = g < groups ? make_int2(a.zero_fill[2 * g], a.zero_fill[2 * g + 1]) : make_int2(0, 0);
        int2 total;
        const int2 sum = block_scan(make_int2(min(max(0, range.y), NvS), 0), s.warp_sum, total);
        if (g < groups) {
          first[g] = range.x;
          cum[g] = pads + sum.x;
        }
        pads += total.x;
      }
      lay = {first, nullptr, nullptr, cum, groups};
      __syncthreads();
    }
    // The phases' times: of the planning from a warp that streams no rows, of the rows from one that does.
    const bool times_plan = tid == kEntries - 32;
    unsigned long long t_laid = 0, t_planned = 0;
    if (times_plan || tid == kEntries) t_laid = globaltimer_ns();
    if (times_plan && a.fresh) stat_phase(c, MOONEP_PH_TABLES, t_begin, t_laid);
    if (warp >= kPlanWarps) {
      clear_pads(c, a, lay, s.grab[warp - kPlanWarps], zeros, shard, meta, epoch);
      if (tid == kEntries) stat_phase(c, MOONEP_PH_ZERO, t_laid);
      if (a.fresh)  // rows behind the last group are unused
        for (int row = used + blockIdx.x * (kThreads - kEntries) + tid - kEntries; row < NvS;
             row += gridDim.x * (kThreads - kEntries)) {
          meta[c.src_info_off + row] = -1;
          if (a.plan_src_info != nullptr) a.plan_src_info[row] = -1;
          if (a.plan_link != nullptr) a.plan_link[row] = 0;
        }
    } else {
      if (t_lo < t_hi) {
        if (a.fresh) {
          plan_tokens(c, a, s, early, cnt, off, cur, meta, before, t_lo, t_hi);
          plan_sync();
          // the release covers what the barrier has ordered before it
          if (tid == kEntries - 32) st_release_gpu(a.work + kWorkReady + blockIdx.x, epoch);
          if (times_plan) stat_phase(c, MOONEP_PH_TOKENS, t_laid);
        } else {
          for (int i = t_lo * K + tid; i < t_hi * K; i += kEntries) {
            const int d = a.dst[i];
            const int loff = d < 0 ? -d - 1 : d;
            if (loff < 0 || loff >= NvS)
              record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_DISPATCH_SEND, 6, d, i / K, i % K);
            else if (a.weights != nullptr)
              reinterpret_cast<float*>(meta + c.weights_off)[loff] = a.weights[i];
          }
        }
      }
      if (tid == 0) t_planned = globaltimer_ns();
      if (!a.bulk)
        copy_plain(c, a, t_lo, t_hi, shard, meta, epoch);
      else if (warp < a.copy_warps) {
        const bool listed = a.fresh && (t_hi - t_lo) * K <= kEntries;  // planned in one step: s.loff still holds them all
        ok = copier.run(reinterpret_cast<unsigned char*>(shard), meta, epoch, t_lo, listed ? t_hi : t_lo);
      }
      // rows behind the last group go into the copy as they are; the warps that do not stream rows see to it
      const int w0 = a.bulk ? a.copy_warps : 0;
      if (a.out != nullptr && a.fresh && warp >= w0)
        copy_tail(c, a, meta, used, NvS, (int)blockIdx.x * (kEntries - 32 * w0) + tid - 32 * w0,
                  (int)gridDim.x * (kEntries - 32 * w0));
    }
    bulk_wait<0>();
    if (tid == 0) {
      const unsigned long long t_end = globaltimer_ns();
      stat_phase(c, MOONEP_PH_SEND, t_planned, t_end);
      stat_phase(c, MOONEP_PH_BUILD_EXPAND, t_begin, t_end);
    }
  }
  // the last CTA resets the counters and publishes what the general kernels' stages publish; the fence covers what the barrier
  // has ordered before it
  ok = __syncthreads_and(ok ? 1 : 0) != 0;
  if (tid == 0) {
    fence_gpu();
    s.last = atomicAdd(c.counters + MOONEP_CTR_DISPATCH_ARRIVE, 1) == (int)gridDim.x - 1;
    fence_gpu();
  }
  __syncthreads();
  if (!s.last) return;
  for (int i = tid; i < (int)gridDim.x; i += kThreads) a.work[kWorkNext + i] = 0;
  if (tid == 0) {
    a.work[kWorkPads] = 0;
    c.counters[MOONEP_CTR_DISPATCH_ARRIVE] = 0;
    if (run && ok && !poisoned(c)) {
      // whoever reads these is on this GPU: one fence for all of them (a release at system scope each held the kernel's end
      // back by several microseconds)
      const int plan_epoch = abs_epoch(c, MOONEP_FLAG_PLAN, a.epoch_plan), tpe_epoch = abs_epoch(c, MOONEP_FLAG_TPE, a.epoch_tpe);
      const int sent_epoch = abs_epoch(c, MOONEP_FLAG_SENT, a.epoch_sent);
      fence_gpu();
      if (a.fresh) {
        st_relaxed_gpu(c.counters + MOONEP_CTR_PLAN_DONE, plan_epoch);
        st_relaxed_sys(flag_ptr(c, 0, MOONEP_FLAG_TPE, 0), tpe_epoch);
        st_relaxed_sys(flag_ptr(c, 0, MOONEP_FLAG_PLAN, 0), plan_epoch);
      }
      st_relaxed_sys(flag_ptr(c, 0, MOONEP_FLAG_SENT, 0), sent_epoch);
    }
  }
}

// ---- combine ---------------------------------------------------------------------------------------------------

constexpr int kCombineThreads = 512;
// At most so many items per warp.  Many short CTAs instead of a resident grid: SMs that are slower to HBM simply run fewer
// of them.  Below that many items for two CTAs per SM a warp takes fewer, so that a small combine still uses every SM.
constexpr int kCombineItems = 4;
constexpr int kCombineLoads = 8;  // 16-byte loads of a lane in flight together: 128 KB per SM with 32 warps

struct CombineArgs {
  const int* dst;           // [N]
  const uint16_t* in_rows;  // [NvS, H]
  const float* in_w;        // [NvS] or null
  uint16_t* out;            // [S, H]
  float* out_w;             // [S, K] or null
  const int* ready;         // optional: per 128-row block of in_rows, see moonep_combine_push
  int ready_expect;
  int vec_ok;
  int items_per_warp;
  int resident;  // the grid is bounded and strides over the items
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

__device__ __forceinline__ int4 pack8(const float* acc) {
  return make_int4((int)pack_bf16(acc[0], acc[1]), (int)pack_bf16(acc[2], acc[3]), (int)pack_bf16(acc[4], acc[5]),
                   (int)pack_bf16(acc[6], acc[7]));
}

// An item is 256 elements (512 bytes) of a token's row; a warp has kItems of them in hand.  Their rows are added in fp32 in
// ascending k and rounded once; a token with one row is copied as it is.  Bound by HBM, hence by the loads in flight: with
// one item in hand a lane has only K of them, so tokens of up to 4, 2 or 1 rows come 2, 4 or 8 items at a time (kItems > 1
// needs K <= kCombineLoads / kItems and 16-byte rows).  One item in hand -> this: S=65536, H=2048, K=1 244 -> 96 us
// (5.6 TB/s), S=4096, H=7168: K=1 61 -> 27, K=2 65 -> 39, K=4 72 -> 57; on one SM, S=1024, H=4096, K=1 724 -> 160.
template <int kItems, bool kVec = true>
__global__ void __launch_bounds__(kCombineThreads, 2) combine_single_kernel(const MoonepDevCtx c, const CombineArgs a) {
  constexpr int kRows = kCombineLoads / kItems;  // rows of an item whose loads are in flight together
  griddep_wait();
  griddep_launch();
  const int failed = ld_volatile(c.status + MOONEP_ST_CODE);  // looked at when the first entries are on their way
  const int lane = threadIdx.x & 31;
  const int K = c.K, H = c.H, NvS = c.NvS;
  const int npieces = (H + 255) / 256;
  const int items = c.S * npieces;  // S * H elements fit the GPU: far below 2^31
  const int step = a.resident ? gridDim.x * (kCombineThreads / 32) : kCombineThreads / 32;
  const int first = a.resident ? blockIdx.x * (kCombineThreads / 32) : blockIdx.x * (kCombineThreads / 32) * a.items_per_warp;
  const int end = a.resident ? items : min(items, first + step * a.items_per_warp);
  // this lane looks up row k of the warp's item j
  const int j_of = kItems > 1 ? lane / kRows : 0, k_of = kItems > 1 ? lane % kRows : lane;
  const bool looks = j_of < kItems && k_of < K;
  int it = first + (threadIdx.x >> 5);
  // The item that this lane looks up, and how far on its next one is: divisions once, not per item (S=16384, H=1024, K=4 28.2 ->
  // 26.9 us).  With one item in hand the registers for it are not there.
  auto token_of = [&](int i) { return (int)((unsigned)i / (unsigned)npieces); };
  int next_tok = token_of(it + j_of * step), next_piece = it + j_of * step - next_tok * npieces;
  const int on_tok = kItems > 1 ? token_of(kItems * step) : 0, on_piece = kItems * step - on_tok * npieces;
  int d_next = looks && it + j_of * step < end ? a.dst[next_tok * K + k_of] : 0;
  if (failed != 0) return;
  for (; it < end; it += kItems * step) {
    const int mine = it + j_of * step;
    const int my_tok = kItems > 1 ? next_tok : token_of(mine), my_piece = kItems > 1 ? next_piece : mine - my_tok * npieces;
    const int d = d_next;
    if constexpr (kItems > 1) {
      next_tok += on_tok;
      next_piece += on_piece;
      if (next_piece >= npieces) {
        next_piece -= npieces;
        ++next_tok;
      }
    } else {
      next_tok = token_of(mine + step);
    }
    d_next = looks && mine + kItems * step < end ? a.dst[next_tok * K + k_of] : 0;  // not a dependent load then
    int row = d < 0 ? -d - 1 : d;
    const bool here = looks && mine < end;
    const bool valid = here && row >= 0 && row < NvS;
    if (here && !valid) record_status(c, MOONEP_STATUS_BAD_INDEX, MOONEP_K_COMBINE_PUSH, 6, d, my_tok, k_of);
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
    if (here && my_piece == 0 && a.in_w != nullptr && a.out_w != nullptr)
      a.out_w[(long long)my_tok * K + k_of] = valid ? a.in_w[row] : 0.f;
    const unsigned rows = __ballot_sync(0xffffffffu, valid);
    const int nvec = H / 8;
    if constexpr (kItems > 1) {
      int4 v[kItems][kRows];
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const int i = __shfl_sync(0xffffffffu, my_piece, j * kRows) * 32 + lane;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const int from = __shfl_sync(0xffffffffu, row, j * kRows + r);
          v[j][r] = make_int4(0, 0, 0, 0);
          if (from >= 0 && i < nvec) v[j][r] = ld16(reinterpret_cast<const int4*>(a.in_rows + (long long)from * H) + i);
        }
      }
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const int tok = __shfl_sync(0xffffffffu, my_tok, j * kRows);
        const int i = __shfl_sync(0xffffffffu, my_piece, j * kRows) * 32 + lane;
        const unsigned have = (rows >> (j * kRows)) & ((1u << kRows) - 1u);
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        int4 only = make_int4(0, 0, 0, 0);
#pragma unroll
        for (int r = 0; r < kRows; ++r)
          if ((have >> r) & 1u) {
            add8(acc, v[j][r]);
            only = v[j][r];
          }
        if (i < nvec && it + j * step < end)
          st16(reinterpret_cast<int4*>(a.out + (long long)tok * H) + i, __popc(have) == 1 ? only : pack8(acc));
      }
    } else if constexpr (kVec) {
      const int i = my_piece * 32 + lane;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      int4 only = make_int4(0, 0, 0, 0);
      for (int k0 = 0; k0 < K; k0 += kRows) {
        int4 v[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const int from = __shfl_sync(0xffffffffu, row, (k0 + r) & 31);
          v[r] = make_int4(0, 0, 0, 0);
          if (k0 + r < K && from >= 0 && i < nvec)
            v[r] = ld16(reinterpret_cast<const int4*>(a.in_rows + (long long)from * H) + i);
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r)
          if (k0 + r < K && ((rows >> (k0 + r)) & 1u)) {
            add8(acc, v[r]);
            only = v[r];
          }
      }
      if (i < nvec) st16(reinterpret_cast<int4*>(a.out + (long long)my_tok * H) + i, __popc(rows) == 1 ? only : pack8(acc));
    } else {
      // element by element, eight loads of a row in flight (a warp per row, one load at a time: S=4096, H=2044, K=4 113 -> 39 us)
      const int e0 = my_piece * 256 + lane;
      float acc[8];
      uint16_t only[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = 0.f, only[q] = 0;
      for (int k = 0; k < K; ++k) {
        const int from = __shfl_sync(0xffffffffu, row, k);
        if (from < 0) continue;
        uint16_t v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = e0 + q * 32 < H ? a.in_rows[(long long)from * H + e0 + q * 32] : 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          acc[q] += __uint_as_float((unsigned)v[q] << 16);
          only[q] = v[q];
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (e0 + q * 32 >= H) continue;
        const __nv_bfloat16 b = __float2bfloat16_rn(acc[q]);
        a.out[(long long)my_tok * H + e0 + q * 32] = __popc(rows) == 1 ? only[q] : *reinterpret_cast<const uint16_t*>(&b);
      }
    }
  }
}

}  // namespace

}  // namespace moonep

using namespace moonep;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

extern "C" int moonep_single_supported(int E, int B, int S, int K) {
  return E <= kMaxGroups && B <= kMaxGroups && (long long)S * K <= kMaxEntries ? 1 : 0;
}

extern "C" int moonep_single_work_words(void) { return kWorkReady + kMaxCtas; }

extern "C" int moonep_dispatch_single(void* ctx, int fresh, int exact, const int* topk, const int* tpe, int* dst, int* cu_seqlens,
                                      int* experts_to_copy, int* zero_fill, int* remote_stats, int* dup_groups,
                                      int* dup_loffs, int* dup_counts, int* plan_src_info, int* plan_link,
                                      const void* hidden, const float* weights, int with_weights, int epoch_tpe,
                                      int epoch_plan, int epoch_sent, int n_ctas, int* work, void* out, float* out_w,
                                      void* stream) {
  auto* h = (HostCtx*)ctx;
  const MoonepDevCtx& c = h->dev;
  if (c.R != 1 || !moonep_single_supported(c.E, c.B, c.S, c.K)) {
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
  a.shard = (uint16_t*)h->hidden_own;
  a.meta = (int*)h->meta_own;
  a.work = work;
  a.out = fresh ? (uint16_t*)out : nullptr;
  a.out_w = fresh ? out_w : nullptr;
  a.weights = weights;
  a.with_weights = with_weights;
  a.fresh = fresh;
  a.exact = exact;
  a.topk_vec = aligned16(topk) ? 1 : 0;
  a.vec_ok = (c.H % 8 == 0 && aligned16(a.out)) ? 1 : 0;
  // MOONEP_EXPAND_PATH=ldst selects register copies as it does with several ranks (S=4096, H=7168, K=8, E=32: 126 us
  // against 112 with bulk copies); looked up once, a lookup per launch costs 0.8 us
  a.bulk_pads = (a.vec_ok && !h->expand_ldst) ? 1 : 0;
  a.bulk = (a.bulk_pads && aligned16(hidden)) ? 1 : 0;
  a.narrow = aligned16(hidden) ? 0 : 1;
  // rows of 16-byte words take any input (the stores, K per load, stay wide); others move in what all addresses allow
  const uintptr_t bits = (uintptr_t)(2ll * c.H) | (uintptr_t)a.out | (uintptr_t)hidden | 16u;
  a.word = a.vec_ok ? 16 : (int)(bits & (~bits + 1));
  a.epoch_tpe = epoch_tpe;
  a.epoch_plan = epoch_plan;
  a.epoch_sent = epoch_sent;
  const size_t static_bytes = sizeof(SingleShared) + 1024;
  const size_t limit = (size_t)imax(0, h->max_smem_optin - (int)static_bytes);
  const size_t tables = (fresh ? (size_t)4 * c.E : (size_t)2 * (c.E + c.B)) * sizeof(int);
  const long long row_bytes = (long long)c.H * 2;
  int grid = imax(1, imin(imin(c.local_sms, h->sm_count), kMaxCtas));
  if (n_ctas > 0) grid = imin(grid, n_ctas);
  a.tokens_per_cta = (c.S + grid - 1) / grid;
  a.stage_bytes = 0;
  a.npieces = a.tokens_per_unit = 1;
  a.copy_warps = 0;
  if (a.bulk) {
    const long long room = (long long)(limit - tables - kZeroBytes);
    const long long most = room / (4 * kRing) / 16 * 16 < kMaxStage ? room / (4 * kRing) / 16 * 16 : kMaxStage;
    a.npieces = (int)((row_bytes + most - 1) / most);
    if (a.npieces > 1) {
      a.stage_bytes = (int)(((row_bytes + a.npieces - 1) / a.npieces + 15) / 16 * 16);
    } else {
      const int share = imax(1, imin(kUnitTokens, (int)(room / (kCopyWarps * kRing) / row_bytes)));
      const int units = kCopyWarps * ((a.tokens_per_cta + kCopyWarps * share - 1) / (kCopyWarps * share));  // as many for each warp
      a.tokens_per_unit = (a.tokens_per_cta + units - 1) / units;
      a.stage_bytes = (int)(a.tokens_per_unit * row_bytes);
    }
    a.copy_warps = imin(kCopyWarps, (int)(room / ((long long)kRing * a.stage_bytes)));
  }
  a.pads_per_grab = imax(1, imin(32, (int)(28672 / row_bytes)));
  const size_t smem = (size_t)a.copy_warps * kRing * a.stage_bytes + (a.bulk_pads ? kZeroBytes : 0) + tables;
  if (!h->single_smem_set) {
    if (int rc = check_cuda(cudaFuncSetAttribute(dispatch_single_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit),
                            "cudaFuncSetAttribute(dispatch_single_kernel)"))
      return rc;
    h->single_smem_set = 1;
  }
  const int per_round = imax(1, a.copy_warps * a.tokens_per_unit), rounds = (a.tokens_per_cta + per_round - 1) / per_round;
  // elsewhere as many as are asked for before the tokens are planned
  a.rounds = rounds <= kDealtRounds && a.tokens_per_cta * (c.K + 1) * row_bytes <= kDealtBytes ? rounds : imin(rounds, kRing - 1);
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
  const long long items = (long long)c.S * ((c.H + 255) / 256);
  a.resident = c.local_sms < h->sm_count ? 1 : 0;
  const long long slots = 2 * kCombineThreads / 32 * (long long)imax(1, a.resident ? c.local_sms : h->sm_count);  // warps at once
  // as many items in hand as fill a lane's loads, as long as every warp slot gets some: below that the latency of one round
  // trip counts and fewer SMs would do the work
  int hand = !a.vec_ok || c.K > 4 ? 1 : c.K > 2 ? 2 : c.K > 1 ? 4 : 8;
  while (hand > 1 && items < hand * slots) hand /= 2;
  a.items_per_warp = hand * (int)(items / (hand * slots) < 1 ? 1 : items / (hand * slots));
  a.items_per_warp = imin(imax(kCombineItems, hand), a.items_per_warp);
  const int per_cta = kCombineThreads / 32 * a.items_per_warp;
  int grid = (int)((items + per_cta - 1) / per_cta);
  if (a.resident) grid = imin(grid, 2 * imax(1, c.local_sms));
  auto* kernel = !a.vec_ok   ? combine_single_kernel<1, false>
                 : hand == 1 ? combine_single_kernel<1>
                 : hand == 2 ? combine_single_kernel<2>
                 : hand == 4 ? combine_single_kernel<4>
                             : combine_single_kernel<8>;
  if (int rc = check_cuda(launch_maybe_pdl(kernel, grid, kCombineThreads, 0, (cudaStream_t)stream, h->enable_pdl != 0, c, a),
                          "launch combine_single_kernel"))
    return rc;
  return check_launch("combine_single_kernel");
}
