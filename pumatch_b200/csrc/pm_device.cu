// pm_device.cu -- device half of libpumatch_b200.so: graph placement, the GPU
// root filter, and the persistent DFS subgraph-enumeration kernel.
//
// Kernel design (sm_100a, 148 SMs):
//   * one persistent grid, sized to the SM count times the resident blocks
//     per SM; every warp runs its own depth-first search;
//   * work = root edges (v0, v1) of one or more plans, handed out in chunks
//     by 64-bit atomic cursors (one per plan, plan after plan);
//   * a warp that still holds a candidate range (at any DFS level) when others
//     have run out of roots cuts its shallowest splittable range and hands the
//     pieces, with the path prefix, to waiting warps by ticket (replaces the
//     reference's disabled stealing, src/gpu_match.cu:21-148, 818-853);
//   * each level's candidate sets ("slots") are read in place where they are
//     an adjacency list or their parent, else computed by a warp-cooperative
//     sorted-set operation -- 64 elements per step, __ballot_sync/__popc
//     compaction -- and stored in a per-warp arena in HBM sized to the plan's
//     worst case, so nothing is truncated (the reference caps every set at
//     GRAPH_DEGREE=4096; that cap is kept only as an explicit emulation
//     switch);
//   * the last level is counted, never materialised: with the level before it
//     in one pass where the plan allows (pair_levels), cliques in bit sets
//     (clique_bits), labeled tails from tables per vertex (chain_kernel), else
//     work-balanced across the warp (leaf_flat), one candidate per lane
//     (leaf_batch) or the last two levels one candidate per lane
//     (lane_subtree).
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "pm_common.h"
#include "pm_device.cuh"
#include "pm_paging.cuh"

namespace pm {
const Plan* plan_of(const pm_plan* h);
}
using namespace pm;

#define CK(call)                                                                         \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return fail(PM_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, \
                  __LINE__);                                                             \
  } while (0)

static constexpr unsigned FULL = 0xffffffffu;

// =====================================================================
// Handles
// =====================================================================

// =====================================================================
// Device helpers
// =====================================================================

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Publication of a donated item: the donor's release store of the slot's
// sequence number orders its item writes before it; the taker's acquire load
// orders its item reads after it.
__device__ __forceinline__ void st_release(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// One value a warp has worked out and may meet again (pair_levels).
struct alignas(16) MemoEntry {
  int32_t x;
  uint32_t tag;   // epoch of the (h0, bound); 0: never written
  int32_t value;  // |N(x) n h0| below the bound
  int32_t len;    // length of x's operand (the reference's scan)
};

struct MatchArgs {
  const uint64_t* rowptr;
  const int32_t* colidx;        // HBM residency
  const uint8_t* labels;
  const int32_t* colidx_lab;    // label-grouped lists (labeled, HBM) or null
  const int32_t* lab_off;       // label group offsets (labeled, HBM or paged) or null
  const int32_t* host_sorted;   // labeled paged: the id-sorted lists in mapped host memory
  int32_t leaf_flat;            // last level: 0 one candidate per lane, 1 flat in lane-contiguous parts,
                                // 2 flat strided (leaf_flat)
  int32_t clique_bits;          // cliques in bit sets
  int32_t memo_entries;         // entries of a warp's value table (a power of two), and the tables: each
  MemoEntry* memo;              // warp's entries, then one that holds the last epoch it used (null: none)
  const unsigned long long* asym;  // two words, 0 when every adjacency entry has its reverse, none comes twice and
                                   // none is its own vertex (maxnbrdeg_kernel)
  const int32_t* hub_slot;      // unlabeled, HBM: [n] bit row of a vertex with a long list, or -1 (null: none)
  const unsigned* hub_bits;     // bit rows of hub_words words: bit u of v's row = u is in v's list
  int32_t hub_words;
  int32_t lane_subtree_max;     // lane_subtree when the parent set is at most this long; 0 = never
  int32_t nl1;
  int32_t n;
  int32_t nplans;
  int32_t T;
  int32_t chunk;                // root edges per shard unit (shard k takes units k, k + count, ...)
  int32_t pop;                  // root edges per queue pop, <= chunk
  int32_t shard_rank;
  int32_t shard_count;
  int32_t split_min;            // donate last-but-one-level ranges at least this long
  int32_t maxdeg;
  unsigned long long* cursors;  // [nplans]
  unsigned long long* counts;   // [nplans]
  unsigned long long* stats;    // [16]
  unsigned int* status;
  int32_t* arena;               // the warps' own arenas
  int64_t arena_words;          // per warp, including the gather space
  int64_t slot_words;           // per warp, slots only (gather space follows)
  int64_t gather_words;         // per warp: space for lists copied out of frames or host memory (paged)
  // Borrowed arenas: a warp whose candidate sets or copied lists outgrow its
  // own arena borrows one of n_big arenas sized for the plans' worst case,
  // for the rest of the root (or donated piece) it is on.
  int32_t* big_arena;
  int64_t big_slot_words;       // per borrowed arena: slots
  int64_t big_gather_words;     // per borrowed arena: gather space after the slots
  unsigned int* big_owner;      // [n_big]: 0 free, 1 held
  int32_t n_big;
  int32_t pad2;
  unsigned long long* root_counts;
  float* root_cost;
  float* root_reads;
  const int32_t* root_order;
  const int32_t* root_split;      // optional per-root donation threshold of the last-but-one level (plan 0)
  // work hand-off (publish_pieces, wait_piece), in don_groups groups of blocks:
  // a warp out of work draws a ticket of its group and waits on the group's
  // ring slot of that number; a warp with work fills the oldest tickets' slots
  // of a group with (plan, root, level, begin, end, path[2..level])
  int4* don_items;                // 3 int4 per slot
  unsigned long long* don_ready;  // per slot: 0 empty, kClaimed being filled, ticket + 1 filled, kQuit no more work
  unsigned long long* sched;      // per group, kSchedStride apart: (tickets drawn << 32) | pieces handed out
  unsigned long long* all_sched;  // the same over all groups
  unsigned int* started;          // warps that have begun
  unsigned int don_groups;        // a power of two; each has kGroupSlots slots
  unsigned int total_warps;
  unsigned long long* heartbeat;  // bumped by busy warps
  unsigned long long timeout_ns;  // hard limit on the launch; idle warps also give
                                  // up after this long without a heartbeat
  DPaging pg;
  // prefetch (paged, plan 0): pages to request for each root chunk, posted
  // when the chunk pf_ahead chunks earlier is claimed (CSR over chunks)
  const int32_t* pf_off;
  const int32_t* pf_pages;
  int32_t pf_ahead;
  int32_t pf_chunks;
  // the launch's plans, in the kernel's own parameter block: every launch
  // carries its own copy, so launches that overlap on a device (other
  // contexts, prepared queries, the allocation-free entry) never see each
  // other's plans
  DPlan plans[PM_MAX_BATCH];
};

// The warps' value tables (pair_levels): kept with the context or the query,
// zeroed when their layout changes -- epochs go on from launch to launch, so
// what an earlier launch left is never taken for a value.
struct MemoTables {
  MemoEntry* d = nullptr;
  size_t bytes = 0;
  int64_t warps = 0;
  int entries = 0;
};

enum { ST_SETOPS = 0, ST_BYTES = 1, ST_ROOTS = 2, ST_SPLITS = 3, ST_HITS = 4, ST_MISSES = 5,
       ST_ZC_BYTES = 6, ST_REQUESTS = 7, ST_EVICTIONS = 8, ST_DROPPED = 9, ST_WARP_NS = 10, ST_IDLE_NS = 11,
       ST_BORROWS = 12, ST_LEAF_CYC = 13, ST_LEVEL_CYC = 14, ST_PREFIX_CYC = 15, ST_PREFETCH = 16,
       ST_DEV_LOADS = 17, ST_DEV_BYTES = 18 };
// control block words: cursors[32] counts[32] stats[kStatWords] status/active ...
constexpr int kStatWords = 24;

#define PM_SB_MAX 512      // ints of a leaf batch's common operand kept in shared memory
#define PM_LANE_MAX 96     // longest first operand one lane handles alone in a leaf batch
#define PM_LEAF_BATCH 512  // candidates per leaf batch

struct alignas(16) WarpState {
  int32_t path[8];
  int32_t iter[8];
  int32_t iend[8];   // exclusive end of the iteration range per level
  int32_t top[9];    // arena offset where level L's slots start
  int32_t size[16];          // members of each slot
  int32_t raw[16];           // elements at ptr: the members and the path vertices among them
  const int32_t* ptr[16];    // each slot's elements: in the arena, or in place in an adjacency array
  unsigned long long id[16]; // names a slot's contents: same name and length, same elements
  unsigned long long next_id;
  unsigned long long sb_id;  // contents the structure in sb was built from (0: none), and what it is
  int32_t sb_len, sb_mode, sb_lo, sb_hi;
  unsigned long long cq_id;  // clique search in bit sets: the set its matrix is over, where, how many rows
  unsigned* cq_rows;
  int32_t cq_n;
  // pair_levels: the warp's value table, the epoch in use and what it stands for
  MemoEntry* memo;
  unsigned long long memo_id;
  uint32_t memo_epoch;
  int32_t memo_len, memo_ub;
  int32_t pair_take;             // candidates the last pass could take, by their lists' lengths (pair_pass)
  int32_t pair_off;              // elements of the first candidate's list that passes have walked already
  int32_t lcnt[32];
  unsigned long long prb[32];    // the candidates' lists laid end to end: where each starts
  int32_t pexcl[33];             // and its offset in the row
  long long next_check;          // SM clock at which to look for waiting warps and at the deadline
  long long began;               // SM clock at the start of the current root or piece
  int32_t checks;                // checks made (the heartbeat is bumped on every 16th)
  unsigned long long t_start;    // %globaltimer at kernel entry (ns)
  int32_t* arena;                // slots of the current path: the warp's own arena or a borrowed one
  int32_t* gather;               // gather space for lists copied out of frames or host memory (paged)
  int64_t cap;                   // slot words at `arena`
  int32_t ghalf;                 // words in each of the two gather halves (first and second operand)
  unsigned long long mul[8];     // per level: how many equal subtrees the search below it stands for
  int32_t big;                   // borrowed arena, or -1
  int32_t split;                 // donation threshold of the last-but-one level for the current root
  // Paged mode: frames pinned for a gather; in HBM: elements whose value is not
  // in the table (pair_levels).  (State for a block of eight warps is kept under
  // a third of 100 KB, so that three blocks leave 156 KB of the SM to L1.)
  union {
    int32_t pins[PM_MAX_LIST_PAGES];
    int32_t queue[64];
  };
  alignas(16) int32_t sb[PM_SB_MAX + 4];  // the common operand (bitmap, filter or sorted copy); +4 for a
                                         // bulk copy that starts up to 3 words before it
  unsigned long long mbar;               // completion barrier of the warp's bulk copies
  uint32_t mphase;                       // its current phase
  unsigned long long lrb[32];       // leaf batches: start of each candidate's first operand in colidx
  int32_t lexcl[33];                // leaf batches: offset of each candidate's operand in the flat layout
};

static_assert(3 * (8 * sizeof(WarpState) + 1024 + 256) <= 100 * 1024, "shared memory of three blocks");

// Per-warp work counters (registers; flushed once at kernel exit).
struct Work {
  unsigned long long setops, bytes, reads, borrows, prefetched;
  unsigned long long leaf_cyc, level_cyc, prefix_cyc;  // SM cycles by phase (lane 0's clock)
  unsigned int err;
  PageCounters pc;
};

// CG: the list may sit in an evictable frame; cg: it does (runtime).
template <bool CG>
__device__ __forceinline__ int32_t ld(const int32_t* p, bool cg = true) {
  if (CG && cg) return __ldcg(p);  // evictable frames are refilled during the launch: skip L1
  return *p;
}

// First index of sorted A[0,len) whose element is >= ub: a 32-ary search,
// one strided probe per lane per round (log32(len) rounds).
template <bool CG>
__device__ __forceinline__ int warp_lower_bound(const int32_t* A, int len, int ub, bool cg = true) {
  const int lane = lane_id();
  int lo = 0, hi = len;
  while (hi - lo > 32) {
    const int step = (hi - lo + 31) >> 5;
    const long long idx = lo + (long long)lane * step;
    const bool lt = idx < hi && ld<CG>(A + idx, cg) < ub;
    const int k = __popc(__ballot_sync(FULL, lt));
    if (k == 0) return lo;
    const int nhi = min(hi, lo + k * step);
    lo = lo + (k - 1) * step + 1;
    hi = nhi;
  }
  const int idx = lo + lane;
  const bool lt = idx < hi && ld<CG>(A + idx, cg) < ub;
  return lo + __popc(__ballot_sync(FULL, lt));
}

// Membership of x in sorted B[0, len) by binary search (per lane).
template <bool CG>
__device__ __forceinline__ bool bsearch_in(const int32_t* B, int len, int x, bool cg = true) {
  int lo = 0, hi = len;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ld<CG>(B + mid, cg) < x) lo = mid + 1; else hi = mid;
  }
  return lo < len && ld<CG>(B + lo, cg) == x;
}

// Adjacency list of v in id order: a slice of colidx in HBM, or resolved
// through the page cache (frame, gathered copy, or host read).  A labeled
// paged graph caches its label-grouped copy, so its whole sorted lists are
// read from host memory.
template <bool PAGED>
__device__ __forceinline__ ListRef adj(const MatchArgs& a, WarpState& S, int v, int32_t* gather, Work& w) {
  const uint64_t b = a.rowptr[v];
  const int len = (int)(a.rowptr[v + 1] - b);
  w.reads++;
  if (!PAGED) return ListRef{a.colidx + b, len, -1};
  if (a.host_sorted) return host_list_copy(a.host_sorted + b, len, gather);
  return paged_list(a.pg, b, len, gather, S.pins, w.pc);
}

// Start (relative to v's list) and length of the label-l part of v's list;
// empty for a label no vertex of the graph carries.
__device__ __forceinline__ int2 label_range(const MatchArgs& a, int v, int l) {
  if (l >= a.nl1 - 1) return make_int2(0, 0);
  const int32_t* o = a.lab_off + (int64_t)v * a.nl1;
  const int s0 = o[l];
  return make_int2(s0, o[l + 1] - s0);
}

// The label-l part of v's list, in id order: from the grouped copy in HBM,
// or through the page cache over the grouped copy.
template <bool PAGED>
__device__ __forceinline__ ListRef adj_label(const MatchArgs& a, WarpState& S, int v, int l, int32_t* gather,
                                             Work& w) {
  const uint64_t b = a.rowptr[v];
  const int2 r = label_range(a, v, l);
  w.reads++;
  if (!PAGED) return ListRef{a.colidx_lab + b + r.x, r.y, -1};
  return paged_list(a.pg, b + (uint64_t)r.x, r.y, gather, S.pins, w.pc);
}

// Operands shorter than this are staged by the lanes' own loads: a bulk
// copy's round trip through the mbarrier costs more than a few loads.
#define PM_BULK_MIN 256

// Stages n <= PM_SB_MAX words of the warp's arena into S.sb with one bulk
// asynchronous copy (cp.async.bulk, completion counted in bytes on the warp's
// mbarrier) and returns where src[0] landed: the copy starts at src rounded
// down to 16 bytes and covers whole 16-byte units, which stay inside the
// arena's allocation (every arena allocation has at least 256 bytes of slack
// after its last word); a slot read in place in an adjacency array is copied
// by the lanes.  The wait is bounded: a copy not complete after
// ~2^20 polls returns src itself (the caller reads B from global memory and
// reports DEV_TIMEOUT).
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __noinline__ const int32_t* stage_bulk(WarpState& S, const int32_t* src, int n) {
  const int lane = lane_id();
  __syncwarp();
  if (lane == 0) S.sb_id = 0;  // the buffer no longer holds the structure built last
  if (n < PM_BULK_MIN || src < S.arena || src >= S.arena + S.cap) {
    __syncwarp();
    for (int i = lane; i < n; i += 32) S.sb[i] = src[i];
    __syncwarp();
    return S.sb;
  }
  const uintptr_t sa = reinterpret_cast<uintptr_t>(src);
  const uintptr_t a0 = sa & ~(uintptr_t)15;
  const int head = (int)((sa - a0) >> 2);
  const uint32_t bytes = (uint32_t)(((head + n) * 4 + 15) & ~15);
  const uint32_t mbar = smem_addr(&S.mbar);
  const uint32_t phase = S.mphase;
  // the lanes' earlier generic writes of the slot (global) and accesses of
  // S.sb (shared) come before the asynchronous proxy's read and write
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(S.sb)),
                 "l"(a0), "r"(bytes), "r"(mbar)
                 : "memory");
  }
  uint32_t done = 0;
  for (int spin = 0; spin < (1 << 20) && !done; spin++) {
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(phase)
        : "memory");
  }
  done = __all_sync(FULL, done);
  __syncwarp();
  if (!done) return src;
  if (lane == 0) S.mphase = phase ^ 1u;
  __syncwarp();
  return S.sb + head;
}

// Borrows a worst-case arena for the rest of the current root: copies the
// live slots [0, live) over (same offsets) and switches the warp to it.  The
// warp's own arena is left as it was, so operands already resolved into it
// stay valid.  Waits, up to the launch deadline, while every borrowed arena
// is held; a holder never waits for another one, so holders always finish.
// False (DEV_ARENA_OVERFLOW without a pool, DEV_TIMEOUT at the deadline) when
// none could be had.  Kept out of line: it is rare, and it must not pull the
// caller's counters out of registers.
__device__ __noinline__ unsigned borrow_arena(const MatchArgs& a, WarpState& S, int64_t live) {
  const int lane = lane_id();
  if (S.big >= 0 || a.n_big == 0) return DEV_ARENA_OVERFLOW;
  int got = -1;
  if (lane == 0) {
    const unsigned start = (unsigned)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) % (unsigned)a.n_big;
    while (got < 0) {
      for (int k = 0; k < a.n_big && got < 0; k++) {
        const int i = (int)((start + (unsigned)k) % (unsigned)a.n_big);
        if (*(volatile unsigned int*)&a.big_owner[i] == 0u && atomicCAS(&a.big_owner[i], 0u, 1u) == 0u) got = i;
      }
      if (got < 0) {
        if (global_ns() - S.t_start > a.timeout_ns) break;
        __nanosleep(2000);
      }
    }
  }
  got = __shfl_sync(FULL, got, 0);
  if (got < 0) return DEV_TIMEOUT;
  int32_t* dst = a.big_arena + (int64_t)got * (a.big_slot_words + a.big_gather_words);
  const int32_t* src = S.arena;
  for (int64_t i = lane; i < live; i += 32) dst[i] = src[i];
  __syncwarp();
  if (lane < 16) {  // slots that live in the arena move with it
    const int32_t* q = S.ptr[lane];
    if (q >= src && q < src + live) S.ptr[lane] = dst + (q - src);
  }
  __syncwarp();
  if (lane == 0) {
    S.arena = dst;
    S.cap = a.big_slot_words;
    S.gather = dst + a.big_slot_words;
    S.ghalf = (int32_t)(a.big_gather_words / 2);
    S.big = got;
  }
  __syncwarp();
  return 0;
}

__device__ __forceinline__ bool borrow(const MatchArgs& a, WarpState& S, int64_t live, Work& w) {
  const unsigned f = borrow_arena(a, S, live);
  w.err |= f;
  w.borrows += f ? 0 : 1;
  return f == 0;
}

// Gives a borrowed arena back (after the warp's writes to it) and returns
// the warp to its own arena.
__device__ __forceinline__ void return_arena(const MatchArgs& a, WarpState& S, int32_t* own) {
  if (S.big < 0) return;
  __syncwarp();
  __threadfence();
  __syncwarp();
  if (lane_id() == 0) {
    atomicExch(&a.big_owner[S.big], 0u);
    S.arena = own;
    S.cap = a.slot_words;
    S.gather = own + a.slot_words;
    S.ghalf = (int32_t)(a.gather_words / 2);
    S.big = -1;
  }
  __syncwarp();
}

// Room for `need` slot words from `top` on, borrowing an arena if the warp's
// own is too small; false (w.err set) when no arena can hold them.
__device__ __forceinline__ bool slot_room(const MatchArgs& a, WarpState& S, int64_t top, int64_t need, Work& w) {
  if (top + need <= S.cap) return true;
  if (!borrow(a, S, top, w)) return false;
  if (top + need <= S.cap) return true;
  w.err |= DEV_ARENA_OVERFLOW;
  return false;
}

// Room for copying a list of `len` words into either gather half (slots
// [0, live) are kept), borrowing an arena if needed.
__device__ __forceinline__ bool gather_room(const MatchArgs& a, WarpState& S, int64_t live, int64_t len, Work& w) {
  if (len <= S.ghalf) return true;
  if (!borrow(a, S, live, w)) return false;
  if (len <= S.ghalf) return true;
  w.err |= DEV_ARENA_OVERFLOW;
  return false;
}

// Bound of slot s at level L from the partial order: the smallest (main
// slot) or largest (helper slot) constrained path vertex; INT_MAX if none.
template <bool LABELED>
__device__ __forceinline__ int slot_bound(const DPlan& P, const WarpState& S, int L, int s) {
  if (LABELED || !P.partial[s]) return INT_MAX;
  const bool is_main = (s == P.level_begin[L]);
  long long ub = is_main ? INT_MAX : -1;
  for (int j = 0; j <= L; j++) {
    if (!(P.partial[s] & (1u << j))) continue;
    const long long v = S.path[j];
    if (is_main) { if (v <= ub) ub = v; }
    else if (ub < v) ub = v;
  }
  return ub == -1 ? INT_MAX : (int)ub;
}

// Membership structures for a second operand B (sorted), built in the warp's
// shared staging buffer (PM_SB_MAX words):
enum : int {
  MEMB_BITMAP = 0,  // max B < 32 * PM_SB_MAX: one bit per id in [0, max B]
  MEMB_FILTER = 1,  // |B| <= PM_FILTER_MAX: a one-hash filter of 32 * PM_SB_MAX bits, then a search of B itself
  MEMB_NONE = 2     // longer: a search of B for every element
};
// At this length a third of the filter's bits are set: two of three searches
// are still spared.
#define PM_FILTER_MAX 8192

struct LeafSet {
  const int32_t* t;
  const int32_t* g;  // B itself (MEMB_FILTER)
  int lenB;
  int lo, hi;        // min and max of B: outside [lo, hi] nothing is a member
};

// Whether x can be a member: exact for the bitmap, what the filter says else.
template <int MODE>
__device__ __forceinline__ bool leaf_maybe(const LeafSet& m, int x) {
  if (x < m.lo || x > m.hi) return false;
  const unsigned f = MODE == MEMB_BITMAP ? (unsigned)x : ((unsigned)x * 0x2545F491u) >> 18;  // 14 bits: the buffer
  return (((const unsigned int*)m.t)[f >> 5] >> (f & 31)) & 1u;
}

template <int MODE>
__device__ __forceinline__ bool leaf_member(const LeafSet& m, int x) {
  return leaf_maybe<MODE>(m, x) && (MODE == MEMB_BITMAP || bsearch_in<false>(m.g, m.lenB, x));
}

// The structure for B (whole warp); returns its mode.  `id` names B's
// contents (WarpState::id; 0: unnamed): a structure built for the same
// contents and length is still in the buffer and is used again -- the parent
// set of a level is the second operand of every candidate of that level.
template <bool CG = false>
__device__ __forceinline__ int leaf_build(WarpState& S, const int32_t* B, int lenB, unsigned long long id, LeafSet& m,
                                          bool cg = true) {
  const int lane = lane_id();
  m.t = S.sb;
  m.g = B;
  m.lenB = lenB;
  if (id && id == S.sb_id && lenB == S.sb_len) {
    m.lo = S.sb_lo;
    m.hi = S.sb_hi;
    return S.sb_mode;
  }
  m.lo = lenB ? ld<CG>(B, cg) : 1;
  m.hi = lenB ? ld<CG>(B + lenB - 1, cg) : 0;
  const int mode = m.hi < 32 * PM_SB_MAX ? MEMB_BITMAP : lenB <= PM_FILTER_MAX ? MEMB_FILTER : MEMB_NONE;
  if (mode == MEMB_NONE) return mode;
  __syncwarp();
  unsigned int* bits = (unsigned int*)S.sb;
  const int words = mode == MEMB_FILTER ? PM_SB_MAX : lenB ? (m.hi >> 5) + 1 : 0;
  for (int i = lane; i < words; i += 32) bits[i] = 0;
  __syncwarp();
  for (int base = 0; base < lenB; base += 128) {  // four loads in flight
    int x[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = base + 32 * q + lane;
      x[q] = i < lenB ? ld<CG>(B + i, cg) : -1;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const unsigned f = mode == MEMB_FILTER ? ((unsigned)x[q] * 0x2545F491u) >> 18 : (unsigned)x[q];
      if (x[q] >= 0) atomicOr(&bits[f >> 5], 1u << (f & 31));
    }
  }
  if (lane == 0) {
    S.sb_id = id;
    S.sb_len = lenB;
    S.sb_mode = mode;
    S.sb_lo = m.lo;
    S.sb_hi = m.hi;
  }
  __syncwarp();
  return mode;
}

// Position of x in sorted A[0, len) (first element >= x), one search per
// group of four lanes (x and len uniform within a group, len 0 = no search):
// five-way steps, so eight searches run side by side in log5(len) round trips.
template <bool CG>
__device__ __forceinline__ int group_lower_bound(const int32_t* A, int len, int x, bool cg = true) {
  const int lane = lane_id();
  const int g4 = lane & 3, sh = lane & ~3;
  int lo = 0, hi = len;
  while (__any_sync(FULL, lo < hi)) {
    const int span = hi - lo;
    const int step = (span + 4) / 5;  // 0 for a finished group
    const int idx = lo + (g4 + 1) * step - 1;
    const bool lt = step > 0 && idx < hi && ld<CG>(A + idx, cg) < x;
    const int k = __popc((__ballot_sync(FULL, lt) >> sh) & 15u);
    if (step > 0) {
      if (k < 4) hi = min(hi, lo + (k + 1) * step - 1);  // the first probe not below x
      lo += k * step;
    }
  }
  return lo;
}

// N searches at once: whether each x[q] is in sorted B[0, len).  The steps
// do not depend on what is found, so the loads of a step are in flight
// together.
template <bool CG, int N>
__device__ __forceinline__ void bsearch_n(const int32_t* B, int len, const int (&x)[N], bool (&in)[N], bool cg) {
  int p[N] = {};
  if (len <= 0) {
#pragma unroll
    for (int q = 0; q < N; q++) in[q] = false;
    return;
  }
  for (int n = len; n > 1;) {
    const int h = n >> 1;
#pragma unroll
    for (int q = 0; q < N; q++)
      if (ld<CG>(B + p[q] + h, cg) <= x[q]) p[q] += h;
    n -= h;
  }
#pragma unroll
  for (int q = 0; q < N; q++) in[q] = in[q] && ld<CG>(B + p[q], cg) == x[q];
}

// The elements of A[0, n) that `keep` leaves (keep(x, in): in[q] comes in as
// "x[q] is an element"), in order: counted, and written to out (unless null)
// up to T of them (T 0: all).  Two loads in flight per lane: with one the warp
// waits a load's latency for every tile of 32, with four the code is so long
// that it waits for its instructions (labeled 5-cycle with a tail on 131,072
// vertices: 4.5 ms with four, 3.8 ms with two).
template <bool CG, class Keep>
__device__ __forceinline__ int compact(const int32_t* A, int n, bool cg, int32_t* out, int T, Keep keep) {
  const int lane = lane_id();
  constexpr int U = 2;
  int cnt = 0;
  for (int base = 0; base < n; base += 32 * U) {
    int x[U];
    bool in[U];
#pragma unroll
    for (int q = 0; q < U; q++) {
      const int i = base + 32 * q + lane;
      in[q] = i < n;
      x[q] = in[q] ? ld<CG>(A + i, cg) : 0;
    }
    keep(x, in);
#pragma unroll
    for (int q = 0; q < U; q++) {
      const unsigned bal = __ballot_sync(FULL, in[q]);
      if (out && in[q]) {
        const int pos = cnt + __popc(bal & lanemask_lt());
        if (!T || pos < T) out[pos] = x[q];
      }
      cnt += __popc(bal);
    }
    if (T && cnt >= T) break;  // the result is the first T survivors
  }
  return cnt;
}

// Whether u in N(v) says v in N(u), and each list holds an element once and
// not its own vertex: an undirected simple graph, as the interface asks for.
// What is taken from one list about the other, from a bit about an element, or
// from a vertex's own list being without it, asks first.
__device__ __forceinline__ bool symmetric(const MatchArgs& a) { return a.asym && (a.asym[0] | a.asym[1]) == 0ull; }

// Whether each list holds an element once: then a list met with a slot of at
// most T elements has at most T of them.
__device__ __forceinline__ bool distinct(const MatchArgs& a) { return a.asym && (a.asym[1] & 1ull) == 0ull; }

// v's bit row (pm_graph::d_hub_bits), or null when its list is short.
__device__ __forceinline__ const unsigned* hub_row(const MatchArgs& a, int v) {
  if (!a.hub_slot || !symmetric(a)) return nullptr;
  const int k = a.hub_slot[v];
  return k < 0 ? nullptr : a.hub_bits + (long long)k * a.hub_words;
}

// Makes slot s the elements [0, raw) at ptr, `size` of them members (the rest
// are path vertices, skipped when the slot is walked).  Lane 0 writes.
__device__ __forceinline__ void set_slot(WarpState& S, int s, const int32_t* ptr, int raw, int size,
                                         unsigned long long id) {
  if (lane_id() == 0) {
    S.ptr[s] = ptr;
    S.raw[s] = raw;
    S.size[s] = size;
    S.id[s] = id;
  }
}

// Name of an adjacency array's part in device memory (its contents never
// change): distinct from the running numbers of slots a warp wrote itself.
__device__ __forceinline__ unsigned long long list_id(const int32_t* p) {
  return (unsigned long long)(uintptr_t)p | (1ull << 63);
}

// ---------------------------------------------------------------------
// One slot of level L for the warp's current path.  Restates compute_set
// (src/gpu_match.cu:238-319) with the operand choice of extend
// (src/gpu_match.cu:409-812).  With `last` returns the count; else fills the
// slot and returns the arena words it took at `top`.
//
// What bounds a level is latency: dependent reads of L2-resident lists.  So
// nothing is copied that can be read where it is: a fresh set is the
// adjacency list itself, cut at its bound, with the path vertices in it
// skipped by whoever walks it (DPlan.hole_ok: only where nothing else reads
// the slot); a copy that removes nothing is its parent.  Intersections test
// two elements per lane at a time against a structure in shared memory that
// the candidates of a level share (leaf_build), or look the shorter operand
// up in the longer when that is 16 times as long.
// Measured (B200), cycles of all warps in levels above the last, the 20-pattern
// labeled batch on an R-MAT graph of 65,536 vertices: 1.4e12 -> 1.0e12; the
// launch 433 -> 309 ms.
// ---------------------------------------------------------------------
template <bool LABELED, bool PAGED>
__device__ int run_slot(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int s, int top, bool last,
                        Work& w) {
  const int lane = lane_id();
  const int kind = P.kind[s];
  const int par = P.parent[s];
  const int vL = S.path[L];
  const int T = a.T;
  const uint32_t mask = P.slot_labels[s];
  // a labeled copy whose parent holds no other labels is its parent
  if (LABELED && kind == SLOT_COPY && L > 1 && !(P.slot_labels[par] & ~mask)) {
    const int len = S.size[par];
    w.setops++;
    w.bytes += 9ull * (unsigned long long)len;  // 4 (|A| + |C|) + |A|
    if (!last) set_slot(S, s, S.ptr[par], len, len, S.id[par]);
    return last ? len : 0;
  }
  ListRef RA, RB{nullptr, 0, -1};
  // one-label masks read only that label's part of an adjacency list: same
  // survivors in the same order, no label gathers (accounting still charges
  // the whole list, as the reference scans it)
  const bool by_label = LABELED && a.lab_off && __popc(mask) == 1 && (kind != SLOT_COPY || L == 1);
  if (PAGED) {
    // the adjacency operands may be copied into the gather halves: make room
    auto list_len = [&](int v) -> int64_t {
      return by_label ? label_range(a, v, __ffs(mask) - 1).y : (int64_t)(a.rowptr[v + 1] - a.rowptr[v]);
    };
    int64_t need = 0;
    if (kind != SLOT_COPY) need = list_len(vL);
    else if (L == 1) need = list_len(S.path[0]);
    if (kind == SLOT_INTERSECT && L == 1) need = max(need, list_len(S.path[0]));
    if (!gather_room(a, S, top, need, w)) {
      if (!last) set_slot(S, s, S.arena + top, 0, 0, 0);
      return 0;
    }
  }
  int32_t* gatherA = S.gather;
  int32_t* gatherB = S.gather + S.ghalf;
  int full_len = -1;  // length of the whole list when by_label
  int full_lenB = -1; // the same for a level-1 second operand read by label (paged)
  unsigned long long idA = 0, idB = 0;
  if (by_label) {
    const int v = (kind != SLOT_COPY) ? vL : S.path[0];
    full_len = (int)(a.rowptr[v + 1] - a.rowptr[v]);
    RA = adj_label<PAGED>(a, S, v, __ffs(mask) - 1, gatherA, w);
  } else if (kind != SLOT_COPY) {
    RA = adj<PAGED>(a, S, vL, gatherA, w);
  } else if (L > 1) {
    RA = ListRef{S.ptr[par], S.size[par], -1};
    idA = S.id[par];
  } else {
    RA = adj<PAGED>(a, S, S.path[0], gatherA, w);
  }
  if (!PAGED && !idA) idA = list_id(RA.p);
  if (kind == SLOT_INTERSECT) {
    if (L > 1) {
      RB = ListRef{S.ptr[par], S.size[par], -1};
      idB = S.id[par];
    } else if (PAGED && by_label) {
      // only the label-l part of N(v0) can meet the label-l part of N(vL)
      const int v0 = S.path[0];
      full_lenB = (int)(a.rowptr[v0 + 1] - a.rowptr[v0]);
      RB = adj_label<PAGED>(a, S, v0, __ffs(mask) - 1, gatherB, w);
    } else {
      RB = adj<PAGED>(a, S, S.path[0], gatherB, w);
      if (!PAGED) idB = list_id(RB.p);
    }
  }
  const int32_t* A = RA.p;
  const int32_t* B = RB.p;
  int lenA = RA.len;
  const int lenB = RB.len;
  const bool cgA = RA.cg, cgB = RB.cg;
  // elements that stay where they are: device memory that outlives the slot
  const bool in_place = !PAGED || (kind == SLOT_COPY && L > 1);
  // each element once, so that leaving a vertex out leaves one element out and
  // an intersection has its elements from either operand
  const bool simple = symmetric(a);

  // symmetry-breaking upper bound (unlabeled only, src/gpu_match.cu:426-458)
  // and, for fresh sets and copies, the path vertices to leave out
  const int ub = slot_bound<LABELED>(P, S, L, s);
  int cnt = 0, used = 0;
  bool done = false;
  if (!LABELED && kind != SLOT_INTERSECT) {
    const int g = lane >> 2;
    const int first = kind == SLOT_FRESH ? 0 : L;  // a copy leaves out the newest vertex only
    const int j = first + g;
    const bool out_v = g < 7 && j <= L;
    const int x = out_v ? S.path[j] : ub;
    const bool search = out_v || (g == 7 && ub != INT_MAX);
    const int pos = group_lower_bound<PAGED>(A, search ? lenA : 0, x, cgA);
    bool hole = out_v && pos < lenA && ld<PAGED>(A + pos, cgA) == x;
    if (hole)
      for (int k = first; k < j; k++) hole = hole && S.path[k] != x;  // one element, left out once
    if (ub != INT_MAX) lenA = __shfl_sync(FULL, pos, 28);
    // a fresh set truncated to T is what remains of the first T elements
    const int scan = (kind == SLOT_FRESH && T && lenA > T) ? T : lenA;
    const int holes = __popc(__ballot_sync(FULL, hole && (lane & 3) == 0 && pos < scan));
    cnt = scan - holes;
    if (!simple) {
      if (last) {
        cnt = compact<PAGED>(A, scan, cgA, nullptr, 0, [&](const int (&v)[2], bool (&in)[2]) {
          for (int k = first; k <= L; k++)
#pragma unroll
            for (int q = 0; q < 2; q++) in[q] = in[q] && v[q] != S.path[k];
        });
        if (T && cnt > T) cnt = T;
        done = true;
      }
    } else if (T && cnt > T) {  // a copy longer than T: its first T survivors
      cnt = T;
      done = last;
      if (in_place && !holes && !last) {
        set_slot(S, s, A, T, T, idA);
        done = true;
      }
    } else if (last) {
      done = true;
    } else if (in_place && (!holes || P.hole_ok[s])) {
      set_slot(S, s, A, scan, cnt, idA);
      done = true;
    }
    if (!done) {
      if (!simple) cnt = T && scan > T ? T : scan;  // room for all of them
      if (slot_room(a, S, top, cnt, w)) {
        int32_t* out = S.arena + top;
        const int want = simple ? cnt : T;
        const int got = compact<PAGED>(A, scan, cgA, out, want, [&](const int (&v)[2], bool (&in)[2]) {
          for (int k = first; k <= L; k++) {
            const int pk = S.path[k];
#pragma unroll
            for (int q = 0; q < 2; q++) in[q] = in[q] && v[q] != pk;
          }
        });
        if (!simple) cnt = T && got > T ? T : got;
      } else {
        cnt = 0;
      }
      used = cnt;
    }
  } else if (LABELED && by_label && kind != SLOT_INTERSECT) {
    cnt = (T && lenA > T) ? T : lenA;
    if (!last) {
      if (in_place) {
        set_slot(S, s, A, cnt, cnt, idA);
        done = true;
      } else {
        if (slot_room(a, S, top, cnt, w))
          compact<PAGED>(A, cnt, cgA, S.arena + top, 0, [](const int (&)[2], bool (&)[2]) {});
        else
          cnt = 0;
        used = cnt;
      }
    }
  } else {
    // labeled by mask, or an intersection
    if (ub != INT_MAX) lenA = warp_lower_bound<PAGED>(A, lenA, ub, cgA);
    const bool check = LABELED && !by_label;
    auto labelled = [&](const int (&v)[2], bool (&in)[2]) {
      if (check) {
#pragma unroll
        for (int q = 0; q < 2; q++) in[q] = in[q] && ((mask >> a.labels[v[q]]) & 1u);
      }
    };
    const unsigned* row = nullptr;
    // (a list that holds an element twice may meet B in more than lenB elements)
    int room = kind == SLOT_INTERSECT && distinct(a) ? min(lenA, lenB) : lenA;
    if (T && room > T) room = T;
    int32_t* out = nullptr;
    bool fits = true;
    if (!last) {
      fits = slot_room(a, S, top, room, w);
      out = S.arena + top;
    }
    if (!fits || room == 0) {
      cnt = 0;
    } else if (kind != SLOT_INTERSECT) {
      cnt = compact<PAGED>(A, lenA, cgA, out, T, labelled);
    } else if (!LABELED && !PAGED && lenB <= lenA && (row = hub_row(a, vL))) {
      // the newest vertex has a bit row: one load per element of the parent
      cnt = compact<PAGED>(B, lenB, cgB, out, T, [&](const int (&v)[2], bool (&in)[2]) {
#pragma unroll
        for (int q = 0; q < 2; q++) in[q] = in[q] && v[q] < ub && ((__ldg(row + (v[q] >> 5)) >> (v[q] & 31)) & 1u);
      });
    } else if (!LABELED && !PAGED && L == 1 && (row = hub_row(a, S.path[0]))) {
      cnt = compact<PAGED>(A, lenA, cgA, out, T, [&](const int (&v)[2], bool (&in)[2]) {
#pragma unroll
        for (int q = 0; q < 2; q++) in[q] = in[q] && ((__ldg(row + (v[q] >> 5)) >> (v[q] & 31)) & 1u);
      });
    } else if ((long long)lenB * 16 < lenA && simple) {
      cnt = compact<PAGED>(B, lenB, cgB, out, T, [&](const int (&v)[2], bool (&in)[2]) {
        bsearch_n<PAGED>(A, lenA, v, in, cgA);
        labelled(v, in);
      });
    } else if ((long long)lenA * 16 < lenB && !(idB && idB == S.sb_id && lenB == S.sb_len)) {
      cnt = compact<PAGED>(A, lenA, cgA, out, T, [&](const int (&v)[2], bool (&in)[2]) {
        bsearch_n<PAGED>(B, lenB, v, in, cgB);
        labelled(v, in);
      });
    } else {
      LeafSet m;
      const int mode = leaf_build<PAGED>(S, B, lenB, idB, m, cgB);
      cnt = compact<PAGED>(A, lenA, cgA, out, T, [&](const int (&v)[2], bool (&in)[2]) {
        if (mode == MEMB_BITMAP) {
#pragma unroll
          for (int q = 0; q < 2; q++) in[q] = in[q] && leaf_maybe<MEMB_BITMAP>(m, v[q]);
        } else {
          if (mode == MEMB_FILTER) {
#pragma unroll
            for (int q = 0; q < 2; q++) in[q] = in[q] && leaf_maybe<MEMB_FILTER>(m, v[q]);
          }
          if (__any_sync(FULL, in[0] || in[1])) bsearch_n<PAGED>(B, lenB, v, in, cgB);
        }
        labelled(v, in);
      });
    }
    if (T && cnt > T) cnt = T;
    if (!last) used = cnt;
  }
  if (!last && !done) {
    __syncwarp();
    unsigned long long id = 0;
    if (lane == 0) id = ++S.next_id;
    set_slot(S, s, S.arena + top, cnt, cnt, id);
  }
  if (PAGED) {
    __syncwarp();
    unpin(a.pg, RA);
    unpin(a.pg, RB);
  }
  const int alenA = by_label ? full_len : lenA;
  const int alenB = full_lenB >= 0 ? full_lenB : lenB;
  w.setops++;
  w.bytes += 4ull * (unsigned long long)(alenA + alenB + cnt) + (LABELED ? (unsigned long long)alenA : 0ull);
  return last ? cnt : used;
}

// run_slot counting only, out of line: for the callers that rarely need it
// (the search's own calls are inlined once; the kernel's code has to stay
// within the instruction cache).  Its counters come back in `t`, so that the
// caller's stay in registers.
template <bool LABELED, bool PAGED>
__device__ __noinline__ int count_slot(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int s, int top,
                                       Work* t) {
  return run_slot<LABELED, PAGED>(a, P, S, L, s, top, true, *t);
}

__device__ __forceinline__ void add_work(Work& w, const Work& t) {
  w.setops += t.setops;
  w.bytes += t.bytes;
  w.reads += t.reads;
  w.borrows += t.borrows;
  w.err |= t.err;
  w.pc.hits += t.pc.hits;
  w.pc.misses += t.pc.misses;
  w.pc.zc_bytes += t.pc.zc_bytes;
  w.pc.requests += t.pc.requests;
  w.pc.evictions += t.pc.evictions;
  w.pc.dropped += t.pc.dropped;
  w.pc.dev_loads += t.pc.dev_loads;
  w.pc.dev_bytes += t.pc.dev_bytes;
}

// A slot equal to, or a prefix of, a slot already computed at this level:
// no scan, only the reference's accounting for the set operation it stands
// for (its first operand's length below its bound, its result length).
template <bool LABELED, bool PAGED>
__device__ void alias_slot(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int s, int live, Work& w) {
  const int t = P.alias[s];
  const int ub = slot_bound<LABELED>(P, S, L, s);
  if (PAGED && ub != INT_MAX) {
    const int v = P.kind[s] != SLOT_COPY ? S.path[L] : S.path[0];
    if ((P.kind[s] != SLOT_COPY || L == 1) && !gather_room(a, S, live, (int64_t)(a.rowptr[v + 1] - a.rowptr[v]), w))
      return;
  }
  int size = S.size[t];
  if (P.alias_prefix[s] && ub != INT_MAX) size = warp_lower_bound<false>(S.ptr[t], size, ub);
  // first operand length as the reference would scan it
  const int kind = P.kind[s];
  int lenA, lenB = 0;
  if (kind != SLOT_COPY) {
    const int v = S.path[L];
    lenA = (int)(a.rowptr[v + 1] - a.rowptr[v]);
    if (ub != INT_MAX) {
      if (PAGED) {
        ListRef r = adj<PAGED>(a, S, v, S.gather, w);
        lenA = warp_lower_bound<PAGED>(r.p, r.len, ub, r.cg);
        __syncwarp();
        unpin(a.pg, r);
      } else {
        lenA = warp_lower_bound<false>(a.colidx + a.rowptr[v], lenA, ub);
      }
    }
  } else if (L > 1) {
    lenA = S.size[P.parent[s]];
    if (ub != INT_MAX) lenA = warp_lower_bound<false>(S.ptr[P.parent[s]], lenA, ub);
  } else {
    const int v = S.path[0];
    lenA = (int)(a.rowptr[v + 1] - a.rowptr[v]);
    if (ub != INT_MAX) {
      if (PAGED) {
        ListRef r = adj<PAGED>(a, S, v, S.gather, w);
        lenA = warp_lower_bound<PAGED>(r.p, r.len, ub, r.cg);
        __syncwarp();
        unpin(a.pg, r);
      } else {
        lenA = warp_lower_bound<false>(a.colidx + a.rowptr[v], lenA, ub);
      }
    }
  }
  if (kind == SLOT_INTERSECT) {
    if (L > 1) lenB = S.size[P.parent[s]];
    else lenB = (int)(a.rowptr[S.path[0] + 1] - a.rowptr[S.path[0]]);
  }
  w.setops++;
  w.bytes += 4ull * (unsigned long long)(lenA + lenB + size) + (LABELED ? (unsigned long long)lenA : 0ull);
  set_slot(S, s, S.ptr[t], size, size, S.id[t]);
}

// Computes every slot of level L; returns the arena top after them.
template <bool LABELED, bool PAGED>
__device__ __forceinline__ int run_level(const MatchArgs& a, const DPlan& P, WarpState& S, int L, Work& w) {
  int top = S.top[L];
  for (int s = P.level_begin[L]; s < P.level_begin[L + 1]; s++) {
    if (P.alias[s] >= 0) continue;
    top += run_slot<LABELED, PAGED>(a, P, S, L, s, top, false, w);
  }
  __syncwarp();
  for (int s = P.level_begin[L]; s < P.level_begin[L + 1]; s++) {
    if (P.alias[s] < 0) continue;
    alias_slot<LABELED, PAGED>(a, P, S, L, s, top, w);
  }
  if (lane_id() == 0) S.top[L + 1] = top;
  __syncwarp();
  return top;
}

// First index of sorted A[0,len) whose element is >= x (one lane).  A list
// wholly below x (the common case for a symmetry-breaking bound) costs one
// load instead of a dependent chain.
template <bool CG = false>
__device__ __forceinline__ int lane_lower_bound(const int32_t* A, int len, int x, bool cg = true) {
  if (len == 0 || ld<CG>(A + len - 1, cg) < x) return len;
  int lo = 0, hi = len - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ld<CG>(A + mid, cg) < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// One lane intersects the part of sorted A[0,deg) below ub with sorted B
// (usually in shared memory), galloping through B; four loads of A in
// flight.  Sets *lenA to the number of elements of A below ub (the
// reference's scan length) and returns the count of members (label-checked
// when LABELED), or -1 when more than `cap` elements would be scanned (the
// caller hands the candidate to the whole warp).
template <bool LABELED, bool CG>
__device__ __forceinline__ int lane_intersect(const int32_t* A, int deg, int ub, const int32_t* B, int lenB,
                                              const uint8_t* labels, uint32_t mask, int* lenA, bool cg,
                                              int cap = PM_LANE_MAX) {
  int k = 0, p = 0, x = 0;
  while (true) {
    if (x >= cap) return -1;
    int v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] = (x + q < deg) ? ld<CG>(A + x + q, cg) : INT_MAX;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int val = v[q];
      if (x + q >= deg || val >= ub) { *lenA = x + q; return k; }
      int lo = p, step = 1;
      while (lo + step < lenB && B[lo + step] < val) { lo += step; step <<= 1; }
      int hi = min(lo + step + 1, lenB);
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (B[mid] < val) lo = mid + 1; else hi = mid;
      }
      p = lo;
      if (p < lenB && B[p] == val && (!LABELED || ((mask >> labels[val]) & 1u))) k++;
      if (p >= lenB) {  // the rest of A is above all of B: only its length matters
        const int r0 = x + q + 1;
        *lenA = r0 + lane_lower_bound<CG>(A + r0, deg - r0, ub, cg);
        return k;
      }
    }
    x += 4;
  }
}

// One lane's contiguous part [t, tend) of a leaf batch's flat layout
// (candidate j's first operand occupies [lexcl[j], lexcl[j+1]) and starts at
// lists[lrb[j]]): members of B, label-checked when LABELED.
template <bool LABELED, int MODE>
__device__ __forceinline__ unsigned leaf_walk(const MatchArgs& a, const WarpState& S, const LeafSet& m,
                                              const int32_t* lists, uint32_t mask, int t, int tend) {
  unsigned k = 0;
  auto test = [&](int x) {
    bool hit = leaf_member<MODE>(m, x);
    if (LABELED && hit) hit = (mask >> a.labels[x]) & 1u;
    k += hit ? 1u : 0u;
  };
  int j = 0;  // the last candidate whose offset is <= t
#pragma unroll
  for (int step = 16; step; step >>= 1)
    if (S.lexcl[j + step] <= t) j += step;
  while (t < tend) {
    const int jbeg = S.lexcl[j];
    const int stop = min(tend, S.lexcl[j + 1]);
    const int32_t* src = lists + S.lrb[j] + (unsigned long long)(t - jbeg);
    const int n = stop - t;
    // scalar up to a 16-byte boundary, then 128-bit loads, four in flight (two, one at the tail)
    int q = min(n, (int)((4 - ((reinterpret_cast<uintptr_t>(src) >> 2) & 3)) & 3));
    for (int u = 0; u < q; u++) test(__ldg(src + u));
    const int4* v = reinterpret_cast<const int4*>(src + q);
    const int nv = (n - q) >> 2;
    int i = 0;
    for (; i + 4 <= nv; i += 4) {
      const int4 a0 = __ldg(v + i), a1 = __ldg(v + i + 1), a2 = __ldg(v + i + 2), a3 = __ldg(v + i + 3);
      test(a0.x); test(a0.y); test(a0.z); test(a0.w);
      test(a1.x); test(a1.y); test(a1.z); test(a1.w);
      test(a2.x); test(a2.y); test(a2.z); test(a2.w);
      test(a3.x); test(a3.y); test(a3.z); test(a3.w);
    }
    for (; i + 2 <= nv; i += 2) {
      const int4 a0 = __ldg(v + i), a1 = __ldg(v + i + 1);
      test(a0.x); test(a0.y); test(a0.z); test(a0.w);
      test(a1.x); test(a1.y); test(a1.z); test(a1.w);
    }
    if (i < nv) {
      const int4 a0 = __ldg(v + i);
      test(a0.x); test(a0.y); test(a0.z); test(a0.w);
    }
    for (q += 4 * nv; q < n; q++) test(__ldg(src + q));
    t = stop;
    j++;
  }
  return k;
}

// A candidate that is a path vertex left standing in its slot (WarpState::raw
// above size): skipped.
__device__ __forceinline__ bool on_path(const WarpState& S, int L, int v) {
  bool on = false;
  for (int j = 0; j <= L; j++) on = on || S.path[j] == v;
  return on;
}

// The last-level intersections of candidates [b, e) with the common operand
// B, work-balanced across the warp: the first operands of 32 candidates (each
// cut at its symmetry-breaking bound, or one label's part of the list when
// `group` >= 0) are laid end to end and split into 32 contiguous parts, one
// per lane.  A lane finds the candidate owning its part's start once and
// walks on through the following lists, four 128-bit loads in flight, testing
// each element against B's structure in shared memory (leaf_build).  Counts
// only.  Truncation needs no care here: B is a slot, at most T long already,
// and the lists hold an element once (the caller asks: distinct).
// Same set operations, counts and accounting as lane_intersect per candidate.
// Batches averaging under 16 elements per lane, and a.leaf_flat == 2, use
// the strided layout instead (element t0 + lane, owner found per element by
// shuffles): it has no per-lane setup per candidate.  Returns false, having
// done nothing, when B is too long for a structure.
template <bool LABELED>
__device__ bool leaf_flat(const MatchArgs& a, WarpState& S, int L, bool holes, const int32_t* cand, int b, int e,
                          const int32_t* B, int lenB, unsigned long long idB, uint32_t mask, int group,
                          int common_ub, bool self_ub, Work& w, unsigned long long* total_cnt) {
  const int lane = lane_id();
  LeafSet m;
  const int mode = leaf_build(S, B, lenB, idB, m);
  if (mode == MEMB_NONE) return false;
  const int32_t* lists = LABELED && group >= 0 ? a.colidx_lab : a.colidx;
  const bool check = LABELED && group < 0;
  unsigned long long cnt = 0, bytes = 0, ops = 0;  // per lane
  for (int base = b; base < e; base += 32) {
    const int i = base + lane;
    const int c = i < e ? cand[i] : 0;
    const bool mine = i < e && !(holes && on_path(S, L, c));
    int lenA = 0;
    unsigned long long rb = 0;
    if (LABELED && group >= 0) {
      if (mine) {
        rb = a.rowptr[c];
        const int deg = (int)(a.rowptr[c + 1] - rb);
        const int2 gr = label_range(a, c, group);
        rb += (unsigned long long)gr.x;
        lenA = gr.y;
        bytes += 4ull * (unsigned long long)(deg + lenB) + (unsigned long long)deg;
        ops++;
      }
    } else if (mine) {
      rb = a.rowptr[c];
      const int deg = (int)(a.rowptr[c + 1] - rb);
      const int ub = self_ub ? min(common_ub, c) : common_ub;
      lenA = (ub == INT_MAX) ? deg : lane_lower_bound(a.colidx + rb, deg, ub);
      bytes += 4ull * (unsigned long long)(lenA + lenB) + (LABELED ? (unsigned long long)lenA : 0ull);
      ops++;
    }
    int incl = lenA;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    // short lists (under 16 elements per lane): the strided layout has no
    // per-candidate setup per lane
    if (a.leaf_flat == 2 || total < 16 * 32) {
      const int excl = incl - lenA;
      for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int j = 0, ej = 0;  // the last lane whose offset is <= t owns element t
#pragma unroll
        for (int step = 16; step; step >>= 1) {
          const int e2 = __shfl_sync(FULL, excl, j + step);
          if (e2 <= t) { j += step; ej = e2; }
        }
        const unsigned long long rbj = __shfl_sync(FULL, rb, j);
        if (t < total) {
          const int x = lists[rbj + (unsigned long long)(t - ej)];
          bool hit = mode == MEMB_BITMAP ? leaf_member<MEMB_BITMAP>(m, x) : leaf_member<MEMB_FILTER>(m, x);
          if (check && hit) hit = (mask >> a.labels[x]) & 1u;
          cnt += hit ? 1u : 0u;
        }
      }
      continue;
    }
    S.lrb[lane] = rb;
    S.lexcl[lane] = incl - lenA;
    if (lane == 31) S.lexcl[32] = total;
    __syncwarp();
    const int chunk = (total + 31) >> 5;
    const int t = min(total, lane * chunk);
    const int tend = min(total, t + chunk);
    unsigned k;
    if (LABELED && check) {
      if (mode == MEMB_BITMAP) k = leaf_walk<true, MEMB_BITMAP>(a, S, m, lists, mask, t, tend);
      else k = leaf_walk<true, MEMB_FILTER>(a, S, m, lists, mask, t, tend);
    } else {
      if (mode == MEMB_BITMAP) k = leaf_walk<false, MEMB_BITMAP>(a, S, m, lists, mask, t, tend);
      else k = leaf_walk<false, MEMB_FILTER>(a, S, m, lists, mask, t, tend);
    }
    cnt += k;
    __syncwarp();
  }
  bytes += 4ull * cnt;  // the results
  for (int o = 16; o; o >>= 1) {
    cnt += __shfl_xor_sync(FULL, cnt, o);
    bytes += __shfl_xor_sync(FULL, bytes, o);
    ops += __shfl_xor_sync(FULL, ops, o);
  }
  w.setops += ops;
  w.bytes += bytes;
  *total_cnt = cnt;
  return true;
}

// The last level for the candidates [b, e) of level L's main slot (each is
// v_{n-2} in turn): one lane per candidate, counting only.  Same set
// operations and counts as run_slot(last) per candidate, organised so that
// short operands cost one lane each:
//   * unlabeled fresh sets and copies are counted with binary searches (the
//     prefix below the bound, minus path vertices found in it);
//   * intersections merge the candidate's list with the common second operand
//     (staged in shared memory when it fits), galloping through it;
//   * a labeled copy is the same for every candidate: counted once;
//   * candidates whose first operand is longer than PM_LANE_MAX go back to the
//     warp-cooperative run_slot.
template <bool LABELED, bool PAGED>
__device__ unsigned long long leaf_batch(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int b, int e,
                                         Work& w) {
  const int lane = lane_id();
  const int s = P.last_slot;
  const int kind = P.kind[s];
  const int Lf = L + 1;
  const int32_t* cand = S.ptr[P.level_begin[L]];
  const bool holes = !LABELED && S.raw[P.level_begin[L]] != S.size[P.level_begin[L]];
  const int par = P.parent[s];
  const int32_t* B = S.ptr[par];  // intersect: second operand; copy: first operand
  const int lenB = S.size[par];
  const uint32_t mask = P.slot_labels[s];
  const int T = a.T;
  unsigned long long cnt_warp = 0;  // uniform across lanes
  if (LABELED && kind == SLOT_COPY) {
    int k = 0;
    for (int i = lane; i < lenB; i += 32) k += (mask >> a.labels[B[i]]) & 1u;
    for (int o = 16; o; o >>= 1) k += __shfl_xor_sync(FULL, k, o);
    if (T && k > T) k = T;
    const unsigned long long m = (unsigned long long)(e - b);
    w.setops += m;
    w.bytes += m * (4ull * (unsigned long long)(lenB + k) + (unsigned long long)lenB);
    return m * (unsigned long long)k;
  }
  // symmetry-breaking bound: bits 0..L are common, bit L+1 is the candidate
  int common_ub = INT_MAX;
  bool self_ub = false;
  if (!LABELED && P.partial[s]) {
    for (int j = 0; j <= L; j++)
      if (P.partial[s] & (1u << j)) common_ub = min(common_ub, S.path[j]);
    self_ub = (P.partial[s] >> Lf) & 1u;
  }
  if (!PAGED && kind == SLOT_INTERSECT && a.leaf_flat && (!T || distinct(a))) {
    const int group = (LABELED && a.lab_off && __popc(mask) == 1) ? __ffs(mask) - 1 : -1;
    unsigned long long k;
    if (leaf_flat<LABELED>(a, S, L, holes, cand, b, e, B, lenB, S.id[par], mask, group, common_ub, self_ub, w, &k))
      return k;
  }
  const unsigned adjacent = !PAGED && symmetric(a) ? P.leaf_adj : 0u;  // path vertices in every candidate's list
  const int32_t* Bs = B;
  if (kind == SLOT_INTERSECT && lenB <= PM_SB_MAX && lenB > 0) {
    Bs = stage_bulk(S, B, lenB);
    if (Bs == B) w.err |= DEV_TIMEOUT;
  }
  unsigned long long cnt = 0, bytes = 0, ops = 0;  // per lane
  PageCounters lpc = {};                           // per lane (paged residency)
  for (int base = b; base < e; base += 32) {
    const int i = base + lane;
    const int c = i < e ? cand[i] : 0;
    const bool mine = i < e && !(holes && on_path(S, L, c));
    bool deferred = false;
    int32_t want = -1;  // an absent page this lane read around, for the warp to load
    if (mine) {
      const int ub = self_ub ? min(common_ub, c) : common_ub;
      if (kind == SLOT_COPY) {  // unlabeled: A = parent slot minus the candidate
        const int lenA = (ub == INT_MAX) ? lenB : lane_lower_bound(B, lenB, ub);
        const int pos = lane_lower_bound(B, lenA, c);
        int k = lenA - ((pos < lenA && B[pos] == c) ? 1 : 0);
        if (T && k > T) k = T;
        cnt += k;
        bytes += 4ull * (unsigned long long)(lenA + k);
        ops++;
      } else {
        const uint64_t rb = a.rowptr[c];
        const int deg = (int)(a.rowptr[c + 1] - rb);
        // a one-label mask reads only that label's part of the list
        const bool grouped = LABELED && a.lab_off && __popc(mask) == 1;
        const int2 gr = grouped ? label_range(a, c, __ffs(mask) - 1) : make_int2(0, deg);
        const int32_t* A = PAGED ? nullptr : (grouped ? a.colidx_lab + rb + gr.x : a.colidx + rb);
        int32_t pinned = -1;
        bool cgl = false;  // A sits in an evictable frame
        if (PAGED) {
          // this lane's own list (or label part) when its one page is
          // resident (pinned and read from the frame) or it spans consecutive
          // static frames; a missing page, a list over evictable pages, or a
          // whole sorted list of a labeled graph (host memory) goes to the
          // warp, which reads host memory coalesced, gathers and requests pages
          const uint64_t s0 = rb + (uint64_t)gr.x;
          const int sh = a.pg.page_shift;
          if (LABELED && !grouped) {
            deferred = true;
          } else if (gr.y == 0) {
            A = a.pg.host_colidx + s0;  // nothing is read
          } else {
            const int32_t p0 = (int32_t)(s0 >> sh);
            const int32_t p1 = (int32_t)((s0 + (uint64_t)gr.y - 1) >> sh);
            const int32_t f = (p0 == p1) ? (pinned = try_pin(a.pg, p0)) : static_run(a.pg, p0, p1);
            if (f >= 0) {
              A = a.pg.frames + ((uint64_t)f << sh) + (s0 & ((1ull << sh) - 1));
              cgl = f >= a.pg.n_static;
              lpc.hits++;
            } else if (p0 == p1 && gr.y <= PM_LANE_MAX) {
              // a short list on a missing page: this lane copies it from host
              // memory into its own part of the gather space, 16 reads in
              // flight per round trip, and notes the page for the warp to
              // load after the batch (or posts it to the host thread)
              if (ld_vol(&a.pg.page_frame[p0]) == PAGE_ABSENT) {
                if (a.pg.dev_copy) want = p0;
                else request_page(a.pg, p0, lpc);
              }
              const int32_t* src = a.pg.host_colidx + s0;
              int32_t* stage = S.gather + lane * PM_LANE_MAX;
              for (int x = 0; x < gr.y; x += 16) {
                int v[16];
#pragma unroll
                for (int q = 0; q < 16; q++) v[q] = (x + q < gr.y) ? src[x + q] : 0;
#pragma unroll
                for (int q = 0; q < 16; q++)
                  if (x + q < gr.y) stage[x + q] = v[q];
              }
              A = stage;
              lpc.misses++;
              lpc.zc_bytes += 4ull * (unsigned long long)gr.y;
            } else {
              deferred = true;
            }
          }
        }
        if (deferred) {
          // handled by the warp below
        } else if (kind == SLOT_INTERSECT && !grouped) {
          int lenA = 0;
          int k = lane_intersect<LABELED, PAGED>(A, deg, ub, Bs, lenB, a.labels, mask, &lenA, cgl);
          if (k < 0) {
            deferred = true;
          } else {
            if (T && k > T) k = T;
            cnt += k;
            bytes += 4ull * (unsigned long long)(lenA + lenB + k) + (LABELED ? (unsigned long long)lenA : 0ull);
            ops++;
          }
        } else {
        const int lenA = (ub == INT_MAX) ? deg : lane_lower_bound<PAGED>(A, deg, ub, cgl);
        if (grouped) {
          // the label-l part of the list: a fresh set is its length, an
          // intersection merges only it
          const int32_t* Al = A;
          const int lenl = gr.y;
          int k = 0;
          if (kind == SLOT_FRESH) {
            k = lenl;
          } else if (lenl > PM_LANE_MAX) {
            deferred = true;
          } else {
            int p = 0;
            for (int x = 0; x < lenl && p < lenB; x++) {
              const int v = ld<PAGED>(Al + x, cgl);
              int lo = p, step = 1;
              while (lo + step < lenB && Bs[lo + step] < v) { lo += step; step <<= 1; }
              int hi = min(lo + step + 1, lenB);
              while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (Bs[mid] < v) lo = mid + 1; else hi = mid;
              }
              p = lo;
              k += (p < lenB && Bs[p] == v) ? 1 : 0;
            }
          }
          if (!deferred) {
            if (T && k > T) k = T;
            cnt += k;
            bytes += 4ull * (unsigned long long)(deg + (kind == SLOT_INTERSECT ? lenB : 0) + k) +
                     (unsigned long long)deg;
            ops++;
          }
        } else if (!LABELED && kind == SLOT_FRESH) {
          // first min(lenA, T) elements, minus the path vertices among them
          const int lim = (T && lenA > T) ? T : lenA;
          // (a path vertex below the bound that the plan made the candidate's
          // neighbour needs no search)
          int k = lim;
          for (int j = 0; j <= L; j++) {
            const int pj = S.path[j];
            if (lim == lenA && ((adjacent >> j) & 1u)) {
              k -= pj < ub ? 1 : 0;
              continue;
            }
            const int pos = lane_lower_bound<PAGED>(A, lim, pj, cgl);
            k -= (pos < lim && ld<PAGED>(A + pos, cgl) == pj) ? 1 : 0;
          }
          cnt += k;
          bytes += 4ull * (unsigned long long)(lenA + k);
          ops++;
        } else if (lenA > PM_LANE_MAX) {
          deferred = true;
        } else if (kind == SLOT_FRESH) {  // labeled: label filter only
          int k = 0;
          for (int x = 0; x < lenA; x++) k += (mask >> a.labels[ld<PAGED>(A + x, cgl)]) & 1u;
          if (T && k > T) k = T;
          cnt += k;
          bytes += 4ull * (unsigned long long)(lenA + k) + (unsigned long long)lenA;
          ops++;
        } else {  // intersection with the common operand
          int k = 0, p = 0;
          for (int x = 0; x < lenA && p < lenB; x++) {
            const int v = ld<PAGED>(A + x, cgl);
            int lo = p, step = 1;
            while (lo + step < lenB && Bs[lo + step] < v) { lo += step; step <<= 1; }
            int hi = min(lo + step + 1, lenB);
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              if (Bs[mid] < v) lo = mid + 1; else hi = mid;
            }
            p = lo;
            if (p < lenB && Bs[p] == v && (!LABELED || ((mask >> a.labels[v]) & 1u))) k++;
          }
          if (T && k > T) k = T;
          cnt += k;
          bytes += 4ull * (unsigned long long)(lenA + lenB + k) + (LABELED ? (unsigned long long)lenA : 0ull);
          ops++;
        }
        }
        if (PAGED && pinned >= 0) unpin_frame(a.pg, pinned);
      }
    }
    // long first operands: the warp takes them one by one
    unsigned dm = __ballot_sync(FULL, deferred);
    while (dm) {
      const int src = __ffs(dm) - 1;
      dm &= dm - 1;
      const int cc = __shfl_sync(FULL, c, src);
      if (lane == 0) S.path[Lf] = cc;
      __syncwarp();
      Work t;
      memset(&t, 0, sizeof(t));
      cnt_warp += (unsigned long long)count_slot<LABELED, PAGED>(a, P, S, Lf, s, S.top[Lf], &t);
      add_work(w, t);
    }
    if (Bs != B && S.sb_id != 0) Bs = stage_bulk(S, B, lenB);  // run_slot built its own structure there
    if (PAGED) {
      // pages the lanes read around: the warp loads up to two of them per
      // 32 candidates (one page copy each), so later reads hit
      unsigned wm = __ballot_sync(FULL, want >= 0);
      for (int k = 0; k < 2 && wm; k++) {
        const int src = __ffs(wm) - 1;
        wm &= wm - 1;
        warp_load_page(a.pg, __shfl_sync(FULL, want, src), w.pc);
      }
    }
  }
  if (PAGED) {
    unsigned long long v[6] = {lpc.hits, lpc.misses, lpc.zc_bytes, lpc.requests, lpc.evictions, lpc.dropped};
#pragma unroll
    for (int k = 0; k < 6; k++)
      for (int o = 16; o; o >>= 1) v[k] += __shfl_xor_sync(FULL, v[k], o);
    w.pc.hits += v[0];
    w.pc.misses += v[1];
    w.pc.zc_bytes += v[2];
    w.pc.requests += v[3];
    w.pc.evictions += v[4];
    w.pc.dropped += v[5];
  }
  for (int o = 16; o; o >>= 1) {
    cnt += __shfl_xor_sync(FULL, cnt, o);
    bytes += __shfl_xor_sync(FULL, bytes, o);
    ops += __shfl_xor_sync(FULL, ops, o);
  }
  w.setops += ops;
  w.bytes += bytes;
  return cnt + cnt_warp;
}

// The last two levels below candidates [b, e) of level L = nnodes-4, one
// lane per candidate v: the lane computes level L+1's intersection X (and
// its alias Y) for path[L+1] = v into its own part of the free arena, then
// counts the last level over X/Y's candidates -- the small sets of light
// subtrees, where warp-wide set operations leave most lanes idle.  Same set
// operations, counts and accounting as run_level + leaf_batch; unlabeled
// plans of the shape DPlan.l2_x describes, X's parent at most lane_subtree_max
// long (it is staged in shared memory); truncation needs no care where the
// lists hold an element once (the caller asks: distinct).  Returns false,
// having counted nothing, when a list that holds an element twice meets the
// parent in more elements than the parent has: a lane's part holds no more.
__device__ bool lane_subtree(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int b, int e, Work& w,
                             unsigned long long* total_cnt) {
  const long long c0 = clock64();
  int32_t* arena = S.arena;
  const int lane = lane_id();
  const int Lq = L + 1;
  const int X = P.l2_x, Y = P.l2_y, M = P.level_begin[Lq], last = P.last_slot;
  const int p1 = P.parent[X];
  const int lenB1 = S.size[p1];
  const int32_t* B1 = S.ptr[p1];
  const int32_t* Bs = lenB1 > 0 ? stage_bulk(S, B1, lenB1) : B1;
  if (lenB1 > 0 && Bs == B1) w.err |= DEV_TIMEOUT;
  const int32_t* cand = S.ptr[P.level_begin[L]];
  const bool holes = S.raw[P.level_begin[L]] != S.size[P.level_begin[L]];
  unsigned long long cnt = 0, bytes = 0, ops = 0;
  bool over = false;
  const int i = b + lane;
  const bool mine = i < e && !(holes && on_path(S, L, cand[i]));
  if (mine) {
    const int v = cand[i];
    // slot bounds with path[Lq] = v: main slots take the smallest constrained
    // path vertex, helpers the largest (slot_bound)
    auto bound = [&](int s) -> int {
      const bool is_main = (s == M);
      long long ub = is_main ? INT_MAX : -1;
      for (int j = 0; j <= Lq; j++) {
        if (!((P.partial[s] >> j) & 1u)) continue;
        const long long pv = (j == Lq) ? v : S.path[j];
        if (is_main) { if (pv <= ub) ub = pv; }
        else if (ub < pv) ub = pv;
      }
      return ub == -1 ? INT_MAX : (int)ub;
    };
    const uint64_t rb = a.rowptr[v];
    const int deg = (int)(a.rowptr[v + 1] - rb);
    const int32_t* A = a.colidx + rb;
    // X = N(v) below its bound, intersected with its parent
    const int ubX = bound(X);
    const int lenAX = (ubX == INT_MAX) ? deg : lane_lower_bound(A, deg, ubX);
    int32_t* buf = arena + S.top[Lq] + lane * lenB1;
    int sizeX = 0, p = 0;
    for (int x = 0; x < lenAX && p < lenB1 && !over; x++) {
      const int val = A[x];
      int lo = p, step = 1;
      while (lo + step < lenB1 && Bs[lo + step] < val) { lo += step; step <<= 1; }
      int hi = min(lo + step + 1, lenB1);
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (Bs[mid] < val) lo = mid + 1; else hi = mid;
      }
      p = lo;
      if (p < lenB1 && Bs[p] == val) {
        over = sizeX == lenB1;
        if (!over) buf[sizeX++] = val;
      }
    }
    bytes += 4ull * (unsigned long long)(lenAX + lenB1 + sizeX);
    ops++;
    // Y: X itself or its prefix below Y's bound, charged as its own operation
    int sizeY = sizeX;
    if (Y >= 0) {
      const int ubY = bound(Y);
      if (P.alias_prefix[Y] && ubY != INT_MAX) sizeY = lane_lower_bound(buf, sizeX, ubY);
      const int lenAY = (ubY == INT_MAX) ? deg : lane_lower_bound(A, deg, ubY);
      bytes += 4ull * (unsigned long long)(lenAY + lenB1 + sizeY);
      ops++;
    }
    const int sizeM = (M == X) ? sizeX : sizeY;
    const int sizeB = (P.parent[last] == X) ? sizeX : sizeY;
    // the last level over the main slot's candidates c
    int common = INT_MAX;
    for (int j = 0; j <= Lq; j++)
      if ((P.partial[last] >> j) & 1u) common = min(common, (j == Lq) ? v : S.path[j]);
    const bool self_ub = (P.partial[last] >> (Lq + 1)) & 1u;
    for (int k = 0; k < sizeM; k++) {
      const int c = buf[k];
      const int ub = self_ub ? min(common, c) : common;
      const uint64_t rc = a.rowptr[c];
      const int dc = (int)(a.rowptr[c + 1] - rc);
      int lenA = 0;
      const int kk = lane_intersect<false, false>(a.colidx + rc, dc, ub, buf, sizeB, a.labels, 0u, &lenA, false,
                                                  INT_MAX);
      cnt += (unsigned long long)kk;
      bytes += 4ull * (unsigned long long)(lenA + sizeB + kk);
      ops++;
    }
  }
  if (__any_sync(FULL, over)) return false;
  w.reads += __popc(__ballot_sync(FULL, mine));  // X's list for each candidate
  for (int o = 16; o; o >>= 1) {
    cnt += __shfl_xor_sync(FULL, cnt, o);
    bytes += __shfl_xor_sync(FULL, bytes, o);
    ops += __shfl_xor_sync(FULL, ops, o);
  }
  w.setops += ops;
  w.bytes += bytes;
  *total_cnt = cnt;
  w.leaf_cyc += (unsigned long long)(clock64() - c0);
  return true;
}

// The rest of a clique search below one node of level L, in bit sets: the
// helper slot of level L (the common neighbours of the path, m of them) is
// numbered, row i of a bit matrix in the arena holds which of them are
// neighbours of number i, and every deeper candidate set is an AND of rows --
// the main set of a candidate is the part of its row below itself, the last
// level is a popcount.  A set operation of the reference's search costs a few
// words instead of a walk over an adjacency list; its operands' lengths are
// known from the rows, two positions per list (len_m: elements below the
// candidate, len_h: elements below the largest path vertex) and the sets'
// sizes, so the accounting is the same.
// Bound: the rows, m^2 / 32 words looked up in the m lists (four searches per
// lane in flight), then L1-resident words.  Measured (B200), 5-clique on an
// R-MAT graph of 32,768 vertices and 524,288 edges: 524 ms with one
// candidate per lane walking its list (lane_subtree), 35 ms so.
#define PM_CLIQUE_MAX 1024  // most common neighbours: 32 words per row, one per lane

__device__ __forceinline__ int64_t clique_words(int m) {
  int wd = 1;
  while (wd * 32 < m) wd <<= 1;
  return 32 + (int64_t)m * (wd + 2);
}

// Bits below number j in word k of a set.
__device__ __forceinline__ unsigned bits_below(int j, int k) {
  const int d = j - 32 * k;
  return d >= 32 ? 0xffffffffu : d <= 0 ? 0u : (1u << d) - 1u;
}

// Rows [0, rows) of the matrix (stride wd words, a power of two) and the two
// lengths of each.  A vertex with a bit row of its own (pm_graph::d_hub_bits)
// answers "is x a neighbour" with one load, 32 numbers a word, eight rows in
// flight; the other lists are short and are scanned -- read in coalesced
// tiles, each element tested against the set's structure in shared memory,
// the few that pass queued and looked up in the set 32 at a time -- or, when
// still much longer than the set, searched for each of its numbers.
// Measured on the 5-clique case above, cycles of all warps in this function:
// searching every row 2.1e11, scanning (hub lists of thousands) 2.1e11, both
// bound by instructions; with bit rows 5.0e10.
#define PM_CLIQUE_SEARCH 448  // list elements per word of the set from which a row is searched

__device__ __noinline__ void clique_rows(const MatchArgs& a, WarpState& S, const int32_t* nb, int m, int wd, int rows,
                                         int ub_h, unsigned long long id, unsigned* R, int32_t* len_m,
                                         int32_t* len_h) {
  const int lane = lane_id();
  const int nw = (m + 31) >> 5;
  int lw = 0;
  while ((1 << lw) < wd) lw++;
  int32_t* queue = (int32_t*)S.lrb;       // 64 words
  unsigned* row_bits = (unsigned*)S.lexcl;  // 32 words
  LeafSet set;
  int mode = MEMB_NONE;  // built when the first row is scanned
  for (int r0 = 0; r0 < rows; r0 += 32) {
    int deg = 0, lh = 0;
    unsigned long long rb = 0;
    if (r0 + lane < rows) {
      const int v = nb[r0 + lane];
      rb = a.rowptr[v];
      deg = (int)(a.rowptr[v + 1] - rb);
      lh = lane_lower_bound(a.colidx + rb, deg, ub_h);
      len_m[r0 + lane] = lane_lower_bound(a.colidx + rb, deg, v);
      len_h[r0 + lane] = lh;
    }
    const int slot = a.hub_slot && r0 + lane < rows ? a.hub_slot[nb[r0 + lane]] : -1;
    const unsigned hubs = __ballot_sync(FULL, slot >= 0);
    if (hubs) {
      const unsigned* bits = a.hub_bits + (long long)max(slot, 0) * a.hub_words;
      for (int k = 0; k < wd; k++) {
        const int x = 32 * k + lane < m ? nb[32 * k + lane] : -1;
        const int at = max(x, 0) >> 5, sh = x & 31;
        for (int r = 0; r < 32; r += 8) {
          if (!((hubs >> r) & 255u)) continue;
          unsigned got[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const unsigned* row = (const unsigned*)__shfl_sync(FULL, (unsigned long long)bits, r + q);
            got[q] = x >= 0 && ((hubs >> (r + q)) & 1u) ? (__ldg(row + at) >> sh) & 1u : 0u;
          }
          unsigned mine = 0;
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const unsigned word = __ballot_sync(FULL, got[q]);
            if (lane == r + q) mine = word;
          }
          if (lane >= r && lane < r + 8 && ((hubs >> lane) & 1u)) R[(r0 + lane) * wd + k] = mine;
        }
      }
    }
    unsigned todo = __ballot_sync(FULL, lh > PM_CLIQUE_SEARCH * nw) & ~hubs;
    const unsigned scans = __ballot_sync(FULL, r0 + lane < rows) & ~todo & ~hubs;
    // searched rows: 8 / wd rows a step, or eight words of one row
    const int per = wd < 8 ? 8 >> lw : 1;
    while (todo) {
      int src[8];
      unsigned left = todo;
#pragma unroll
      for (int q = 0; q < 8; q++) src[q] = -1;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        if (k >= per || !left) continue;
        const int r = __ffs(left) - 1;
        left &= left - 1;
#pragma unroll
        for (int q = 0; q < 8; q++)
          if ((wd < 8 ? q >> lw : 0) == k) src[q] = r;
      }
      todo = left;
      for (int k0 = 0; k0 < wd; k0 += 8) {
        const int32_t* A[8];
        int n[8], x[8], most = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const int k = wd < 8 ? q & (wd - 1) : k0 + q;
          A[q] = a.colidx + __shfl_sync(FULL, rb, src[q] & 31);
          n[q] = src[q] >= 0 ? __shfl_sync(FULL, lh, src[q] & 31) : 0;
          most = max(most, n[q]);
          x[q] = n[q] > 0 && 32 * k + lane < m ? nb[32 * k + lane] : -1;
          if (n[q] == 0) A[q] = nb;  // something readable
        }
        while (most > 1) {
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const int h = n[q] >> 1;
            if (A[q][h] <= x[q]) A[q] += h;
            n[q] -= h;
          }
          most -= most >> 1;
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const unsigned word = __ballot_sync(FULL, x[q] >= 0 && *A[q] == x[q]);
          const int k = wd < 8 ? q & (wd - 1) : k0 + q;
          if (lane == 0 && src[q] >= 0 && k < wd) R[(r0 + src[q]) * wd + k] = word;
        }
      }
    }
    if (scans && mode == MEMB_NONE) mode = leaf_build(S, nb, m, id, set);
    for (unsigned left = scans; left; left &= left - 1) {
      const int r = __ffs(left) - 1;
      const int32_t* A = a.colidx + __shfl_sync(FULL, rb, r);
      const int len = __shfl_sync(FULL, lh, r);
      int queued = 0;
      row_bits[lane] = 0u;
      __syncwarp();
      auto place = [&](int count) {  // the queue's first `count` (at most 32)
        const int x = lane < count ? queue[lane] : -1;
        int at = 0;
        for (int n = m; n > 1;) {
          const int h = n >> 1;
          if (nb[at + h] <= x) at += h;
          n -= h;
        }
        if (x >= 0 && nb[at] == x) atomicOr(&row_bits[at >> 5], 1u << (at & 31));
      };
      for (int base = 0; base < len; base += 128) {
        int x[4];
        bool in[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int i = base + 32 * q + lane;
          in[q] = i < len;
          x[q] = in[q] ? A[i] : 0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
          in[q] = in[q] && (mode == MEMB_BITMAP ? leaf_maybe<MEMB_BITMAP>(set, x[q]) : leaf_maybe<MEMB_FILTER>(set, x[q]));
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const unsigned bal = __ballot_sync(FULL, in[q]);
          if (in[q]) queue[queued + __popc(bal & lanemask_lt())] = x[q];
          queued += __popc(bal);
          __syncwarp();
          if (queued >= 32) {
            place(32);
            __syncwarp();
            const int rest = lane < queued - 32 ? queue[32 + lane] : 0;
            __syncwarp();
            queued -= 32;
            if (lane < queued) queue[lane] = rest;
            __syncwarp();
          }
        }
      }
      if (queued) place(queued);
      __syncwarp();
      if (lane < wd) R[(r0 + r) * wd + lane] = row_bits[lane];
      __syncwarp();
    }
  }
  __syncwarp();
}

// Candidates [b, e) of level L's main slot (the first numbers of the helper
// slot's): matches below them.
__device__ __noinline__ unsigned long long clique_bits(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int b,
                                                       int e, unsigned long long* ops_out,
                                                       unsigned long long* bytes_out,
                                                       unsigned long long* reads_out) {
  const int lane = lane_id();
  const int hs = P.level_begin[L] + 1;
  const int32_t* nb = S.ptr[hs];
  const int m = S.size[hs];
  int wd = 1;
  while (wd * 32 < m) wd <<= 1;
  unsigned* R = (unsigned*)(S.arena + ((S.top[L + 1] + 31) & ~31));
  int32_t* len_m = (int32_t*)(R + m * wd);
  int32_t* len_h = len_m + m;
  if (S.cq_id != S.id[hs] || S.cq_rows != R || S.cq_n < e) {
    int ub_h = 0;
    for (int j = 0; j <= L; j++) ub_h = max(ub_h, S.path[j]);
    const int rows = S.iend[L];
    __syncwarp();
    clique_rows(a, S, nb, m, wd, rows, ub_h, S.id[hs], R, len_m, len_h);
    if (lane == 0) {
      S.cq_id = S.id[hs];
      S.cq_rows = R;
      S.cq_n = rows;
      S.sb_id = 0;
    }
    __syncwarp();
  }
  const int depth = P.nnodes - 4 - L;  // levels between the candidates' and the last
  unsigned long long cnt = 0, ops = 0, bytes = 0;  // per lane
  unsigned reads = 0;  // nodes entered: the level-by-level search reads a list for each
  if (m <= 32) {
    // one candidate per lane, every set one word
    unsigned* rs = (unsigned*)S.sb;
    int32_t* lm = S.sb + 32;
    int32_t* lh = S.sb + 64;
    if (lane == 0) S.sb_id = 0;
    for (int i = lane; i < e; i += 32) {
      rs[i] = R[i];
      lm[i] = len_m[i];
      lh[i] = len_h[i];
    }
    __syncwarp();
    const int i = b + lane;
    if (i < e) {
      unsigned H[3], M[3];
      int d = 0;
      H[0] = rs[i];
      M[0] = H[0] & bits_below(i, 0);
      auto node = [&](int v, int size_up, unsigned h, unsigned mm) {  // the two set operations of a level
        const int nh = __popc(h), nm = __popc(mm);
        ops += 2;
        reads++;
        bytes += 4ull * (unsigned long long)(lm[v] + lh[v] + 2 * size_up + nh + nm);
      };
      node(i, m, H[0], M[0]);
      while (d >= 0) {
        // (depth at most 2: selects instead of indexed registers)
        const unsigned h = d == 0 ? H[0] : d == 1 ? H[1] : H[2];
        unsigned mm = d == 0 ? M[0] : d == 1 ? M[1] : M[2];
        if (d == depth) {
          const int nh = __popc(h);
          while (mm) {
            const int j = __ffs(mm) - 1;
            mm &= mm - 1;
            const int k = __popc(rs[j] & h & bits_below(j, 0));
            cnt += k;
            ops++;
            bytes += 4ull * (unsigned long long)(lm[j] + nh + k);
          }
          d--;
          continue;
        }
        if (!mm) {
          d--;
          continue;
        }
        const int j = __ffs(mm) - 1;
        mm &= mm - 1;
        if (d == 0) M[0] = mm; else M[1] = mm;
        const unsigned h2 = h & rs[j], m2 = h2 & bits_below(j, 0);
        node(j, __popc(h), h2, m2);
        d++;
        if (d == 1) { H[1] = h2; M[1] = m2; } else { H[2] = h2; M[2] = m2; }
      }
    }
    __syncwarp();
  } else {
    // one candidate at a time, word `lane` of every set in lane `lane`; the
    // last level takes 32 / wd candidates a step, wd lanes each
    unsigned short* lst = (unsigned short*)S.sb;
    if (lane == 0) S.sb_id = 0;
    const int grp = lane / wd, gw = lane & (wd - 1), groups = 32 / wd;
    for (int i = b; i < e; i++) {
      unsigned H[3], M[3];
      int size[3];
      int d = 0, v = i;
      unsigned up = lane < ((m + 31) >> 5) ? 0xffffffffu : 0u;  // level L's helper set (all numbers)
      int size_up = m;
      bool fresh = true;  // v was chosen: its sets are to be computed at depth d
      while (d >= 0) {
        if (fresh) {
          const unsigned row = lane < wd ? R[v * wd + lane] : 0u;
          const unsigned h = row & up, mm = h & bits_below(v, lane);
          const int nh = __reduce_add_sync(FULL, __popc(h)), nm = __reduce_add_sync(FULL, __popc(mm));
          if (d == 0) { H[0] = h; M[0] = mm; size[0] = nh; }
          else if (d == 1) { H[1] = h; M[1] = mm; size[1] = nh; }
          else { H[2] = h; M[2] = mm; size[2] = nh; }
          if (lane == 0) {
            ops += 2;
            reads++;
            bytes += 4ull * (unsigned long long)(len_m[v] + len_h[v] + 2 * size_up + nh + nm);
          }
          fresh = false;
        }
        const unsigned h = d == 0 ? H[0] : d == 1 ? H[1] : H[2];
        const unsigned mm = d == 0 ? M[0] : d == 1 ? M[1] : M[2];
        const int nh = d == 0 ? size[0] : d == 1 ? size[1] : size[2];
        if (d == depth) {
          // the main set's numbers, listed in shared memory
          int incl = __popc(mm);
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
          }
          const int total = __shfl_sync(FULL, incl, 31);
          __syncwarp();
          {
            int at = incl - __popc(mm);
            unsigned left = mm;
            while (left) {
              lst[at++] = (unsigned short)(32 * lane + __ffs(left) - 1);
              left &= left - 1;
            }
          }
          __syncwarp();
          const unsigned hw = __shfl_sync(FULL, h, gw);
          unsigned k = 0;
          for (int t = grp; t < total; t += 4 * groups) {
            unsigned r4[4];
            int j4[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const bool on = t + q * groups < total;
              j4[q] = on ? lst[t + q * groups] : 0;
              r4[q] = on ? R[j4[q] * wd + gw] : 0u;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) k += __popc(r4[q] & hw & bits_below(j4[q], gw));
          }
          cnt += k;
          bytes += 4ull * k;
          for (int t = lane; t < total; t += 32) bytes += 4ull * (unsigned long long)(len_m[lst[t]] + nh);
          if (lane == 0) ops += (unsigned long long)total;
          __syncwarp();
          d--;
        } else {
          const unsigned any = __ballot_sync(FULL, mm != 0u);
          if (!any) {
            d--;
          } else {
            const int src = __ffs(any) - 1;
            const int bit = __ffs(__shfl_sync(FULL, mm, src)) - 1;
            v = 32 * src + bit;
            const unsigned left = lane == src ? mm & (mm - 1) : mm;
            if (d == 0) M[0] = left; else M[1] = left;
            up = h;
            size_up = nh;
            d++;
            fresh = true;
          }
        }
        // back at a shallower level: its own helper set is `up` again when
        // the next candidate there is entered (set above)
      }
    }
  }
  for (int o = 16; o; o >>= 1) {
    cnt += __shfl_xor_sync(FULL, cnt, o);
    bytes += __shfl_xor_sync(FULL, bytes, o);
    ops += __shfl_xor_sync(FULL, ops, o);
  }
  *ops_out = ops;
  *bytes_out = bytes;
  *reads_out = __reduce_add_sync(FULL, reads);
  return cnt;
}

// ---------------------------------------------------------------------
// The last two levels in one pass.  Level q = n-3's main slot is a list of
// each candidate v for path[q] (N(v), or its part in a parent slot), and the
// last level adds a value f(x) for every element x of it:
//   PAIR_COPY   the last slot is a copy of a set h of level q (itself a copy
//               of h0, a slot of level q-1): |h|, less one if x is in h;
//   PAIR_FRESH  x's own list: its length (below a bound of the path), less
//               the path vertices in it;
//   PAIR_MEET   x's list intersected with h: |N(x) n h0|, less one when v is
//               in h0 (v is a neighbour of x).  The value depends on x and h0
//               only, and the same x is met under many v: each warp keeps the
//               values in a table of its own in device memory (MemoEntry),
//               tagged with the number of the (h0, bound) they belong to.
//   PAIR_SHARED the main slot itself is a copy of a set s of level q-1, less v,
//               and the last level fresh (unlabeled): the elements are the same
//               for every v but for v itself and its neighbours in s, so the
//               sum over s is taken once, and of each v's list only its members
//               of s are counted -- by the list or, when v has a bit row and s
//               is shorter, by looking s up in the row.
// So no slot of level q is built, and no call is made per candidate of level
// q: the lists of 32 candidates are laid end to end and their elements taken
// 64 at a time, two per lane in flight (a tile per list left most lanes
// without one: the 6-cycle's lists have about ten elements below their bound).
// Each kind is a function of its own: what the loop waits for most is its own
// instructions (no_instruction 9.2 of 25 stall cycles per issue; four elements
// per lane in flight: 6-cycle shard 40 ms, 20-pattern batch 19.2 ms; two: 36.6
// and 16.0; one: 40.9 and 14.9, but the 7-cycle 74 ms for 66).
// Set operations, counts and accounting are those of run_level + leaf_batch.
//
// What bounded the search before was instructions, not bytes: about 1,400 per
// candidate of level q for two slots and a batch whose lists have a few tens
// of elements (house on 3,000 vertices: 2.3 million candidates, 3.2e9 warp
// instructions, 7.4 ms), and for cycles the walk over every list again under
// every v.  Measured (B200), launch before and after: house on 3,000 vertices
// 6.5 -> 1.7 ms; one of 64 shards of the 6-cycle on Chung-Lu 20,000 / 100,000
// 372 -> 68 ms; labeled on R-MAT, the 5-cycle (8 labels, 32,768 vertices, sets
// capped at 4,096) 37 -> 5.3 ms, the 5-cycle with a tail (32 labels, 131,072
// vertices) 18 -> 12.6 ms, paged 47 -> 27 ms.
// ---------------------------------------------------------------------
// Counters of one pass (per lane).
struct PairSums {
  unsigned long long cnt, bytes, elems;
};

// Queued elements whose PAIR_MEET value is not in the table: the first
// `count` (at most 32) of S.queue.  Their lists, cut at the bound or to one
// label's part, are laid end to end and walked in equal parts, a part at a
// time per lane, matches added to the owner's counter in shared memory.
template <bool LABELED>
__device__ __noinline__ void meet_values(const MatchArgs& a, WarpState& S, const LeafSet& m, int mode, int group,
                                            int ub, int count, PairSums& r) {
  const int lane = lane_id();
  const int32_t* lists = LABELED ? a.colidx_lab : a.colidx;
  int lenA = 0, scan_len = 0, x = -1;
  unsigned long long rb = 0;
  if (lane < count) {
    x = S.queue[lane];
    rb = a.rowptr[x];
    const int deg = (int)(a.rowptr[x + 1] - rb);
    if (LABELED) {
      const int2 gr = label_range(a, x, group);
      rb += (unsigned long long)gr.x;
      lenA = gr.y;
      scan_len = deg;
    } else {
      lenA = ub == INT_MAX ? deg : lane_lower_bound(a.colidx + rb, deg, ub);
      scan_len = lenA;
    }
  }
  int incl = lenA;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  S.lrb[lane] = rb;
  S.lexcl[lane] = incl - lenA;
  if (lane == 31) S.lexcl[32] = total;
  S.lcnt[lane] = 0;
  __syncwarp();
  for (int t0 = 0; t0 < total; t0 += 64) {
    int y[2], own[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int t = t0 + 32 * q + lane;
      int j = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1)
        if (S.lexcl[j + step] <= t) j += step;
      own[q] = j;
      y[q] = t < total ? __ldg(lists + S.lrb[j] + (unsigned long long)(t - S.lexcl[j])) : -1;
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const bool hit = y[q] >= 0 && (mode == MEMB_BITMAP ? leaf_member<MEMB_BITMAP>(m, y[q])
                                                          : leaf_member<MEMB_FILTER>(m, y[q]));
      if (hit) atomicAdd(&S.lcnt[own[q]], 1);
    }
  }
  __syncwarp();
  if (lane < count) {
    const int k = S.lcnt[lane];
    r.cnt += (unsigned long long)k;
    r.bytes += 4ull * (unsigned long long)(scan_len + k) + (LABELED ? (unsigned long long)scan_len : 0ull);
  }
  // one lane per table entry stores
  const int at = x & (a.memo_entries - 1);
  const unsigned same = __match_any_sync(FULL, lane < count ? at : -1 - lane);
  if (lane < count && (same & lanemask_lt()) == 0)
    *reinterpret_cast<int4*>(S.memo + at) = make_int4(x, (int)S.memo_epoch, S.lcnt[lane], scan_len);
  __syncwarp();
}

// True when this node's last two levels can be taken in one pass (DPlan.pair:
// the launch's part of the answer).
template <bool LABELED, bool PAGED>
__device__ __forceinline__ bool pair_ready(const MatchArgs& a, const DPlan& P, const WarpState& S) {
  // (a labeled list that holds an element twice may meet a truncated slot in
  // more than T elements)
  if (!P.pair || (LABELED ? a.T && !distinct(a) : !symmetric(a))) return false;
  if (P.pair == PAIR_MEET) {
    const int n0 = S.size[P.pair_h0];
    return n0 <= PM_FILTER_MAX || (n0 > 0 && S.ptr[P.pair_h0][n0 - 1] < 32 * PM_SB_MAX);
  }
  if (P.kind[P.level_begin[P.nnodes - 3]] == SLOT_INTERSECT || P.pair == PAIR_SHARED) {
    const int par = P.parent[P.level_begin[P.nnodes - 3]], n0 = S.size[par];
    return (n0 <= PM_FILTER_MAX || (n0 > 0 && S.ptr[par][n0 - 1] < 32 * PM_SB_MAX));
  }
  return true;
}

// Elements a pass walks at most: the lists of as many of its 32 candidates as
// have this many together, or this much of one list.  A warp looks for waiting
// warps and at the deadline between passes; with no such bound one over 32
// hubs' lists took 19 ms (a 5-path on an R-MAT graph of 262,144 vertices), or
// 136 ms where each element's list is walked in turn (the 5-cycle with 4
// labels); with it 3 and 15 ms.  Labeled, those take half as many (4,096: 27
// ms); unlabeled, half as many cost the 6-cycle shard 8% (38.1 -> 41 ms).  A
// look from inside the walks instead cost the 20-pattern batch 5%; this costs
// it 3% (19.2 -> 19.7 ms).
constexpr int kPairRow = 4096;

template <int N>
__device__ __forceinline__ bool any_of(const bool (&in)[N]) {
  bool any = false;
#pragma unroll
  for (int q = 0; q < N; q++) any = any || in[q];
  return any;
}

// Candidates [b, e) (at most 32) of level L = n-4's main slot, or the first of
// them, or a part of the first one's list; with off > 0 the rest of b's list
// from there, b's own operations counted before.  S.iter[L] and S.pair_off say
// where the next pass goes on.
template <bool LABELED, bool PAGED, int KIND, bool MET>
__device__ __noinline__ unsigned long long pair_pass(const MatchArgs& a, const DPlan& P, WarpState& S, int L, int b,
                                                     int e, int off, Work* wt) {
  Work& w = *wt;
  const int lane = lane_id();
  const int q = L + 1;
  const int ms = P.level_begin[q], last = P.last_slot;
  constexpr int kind = KIND;
  constexpr bool meet_main = MET;  // the main slot is an intersection
  const int main_group = LABELED ? __ffs(P.slot_labels[ms]) - 1 : -1;
  const int last_group = LABELED ? __ffs(P.slot_labels[last]) - 1 : -1;
  // the parent a main intersection meets, and the set a copy or a meeting reads
  LeafSet set;
  int mode = MEMB_NONE;
  int lenBm = 0;
  if (meet_main) {
    const int par = P.parent[ms];
    lenBm = S.size[par];
    mode = leaf_build(S, S.ptr[par], lenBm, S.id[par], set);
  }
  const int h0 = P.pair_h0;
  constexpr bool has_h = KIND == PAIR_COPY || KIND == PAIR_MEET;
  const int32_t* H0 = has_h ? S.ptr[h0] : nullptr;
  const int len0 = has_h ? S.size[h0] : 0;
  // the last slot's bound (a main slot: the smallest constrained path vertex; up to L only in these plans)
  int ub_last = INT_MAX;
  if (!LABELED)
    for (int j = 0; j <= L; j++)
      if ((P.partial[last] >> j) & 1u) ub_last = min(ub_last, S.path[j]);
  int len_h = len0;  // h0 below h's bound (a helper slot: the largest constrained path vertex)
  if (kind == PAIR_MEET) {
    const int ub_h = slot_bound<LABELED>(P, S, L, P.parent[last]);
    if (!LABELED && ub_h != INT_MAX) len_h = warp_lower_bound<false>(H0, len0, ub_h);
    mode = leaf_build(S, H0, len_h, S.id[h0], set);
    if (S.memo_id != S.id[h0] || S.memo_len != len_h || S.memo_ub != ub_last) {
      __syncwarp();
      if (S.memo_epoch == 0xffffffffu) {  // numbers used up: forget everything
        for (int i = lane; i < a.memo_entries; i += 32) *reinterpret_cast<int4*>(S.memo + i) = make_int4(0, 0, 0, 0);
        __syncwarp();
        if (lane == 0) S.memo_epoch = 0;
        __syncwarp();
      }
      if (lane == 0) {
        S.memo_id = S.id[h0];
        S.memo_len = len_h;
        S.memo_ub = ub_last;
        S.memo_epoch++;
      }
      __syncwarp();
    }
  }
  const unsigned epoch = S.memo_epoch;
  // the candidates, one per lane
  const int32_t* cand = S.ptr[P.level_begin[L]];
  const bool holes = !LABELED && S.raw[P.level_begin[L]] != S.size[P.level_begin[L]];
  const int v = b + lane < e ? cand[b + lane] : -1;
  bool mine = v >= 0 && !(holes && on_path(S, L, v));
  unsigned long long rb = 0;
  int len = 0;     // elements of v's list to look at
  int h_v = 0;     // |h| under v (a copy's or a meeting's second operand)
  int less = 0;    // PAIR_MEET: 1 when v is in h0 below the bound
  PairSums r = {0, 0, 0};
  unsigned long long ops = 0;
  if (mine) {
    rb = a.rowptr[v];
    const int deg = (int)(a.rowptr[v + 1] - rb);
    int lenA = deg;
    len = deg;
    if (LABELED) {
      const int2 gr = label_range(a, v, main_group);
      rb += (unsigned long long)gr.x;
      len = gr.y;
    } else if (P.partial[ms]) {
      int ub = INT_MAX;  // a main slot: the smallest constrained path vertex, v among them
      for (int j = 0; j <= L; j++)
        if ((P.partial[ms] >> j) & 1u) ub = min(ub, S.path[j]);
      if ((P.partial[ms] >> q) & 1u) ub = min(ub, v);
      if (ub != INT_MAX) lenA = len = lane_lower_bound(a.colidx + rb, deg, ub);
    }
    // a fresh set holds at most its first T elements; what is made of slots is
    // no longer than they are
    if (a.T && !meet_main) len = min(len, a.T);
    ops = 1;
    if (KIND != PAIR_SHARED)
      r.bytes += 4ull * (unsigned long long)(lenA + lenBm) + (LABELED ? (unsigned long long)lenA : 0ull);
    if (has_h) {
      // h: h0 without v (labeled: h0 itself), below h's bound
      bool in0 = false;
      if (!LABELED) {
        const int at = lane_lower_bound(H0, len_h, v);
        in0 = at < len_h && H0[at] == v;
      }
      h_v = len_h - (in0 ? 1 : 0);
      less = in0 && v < ub_last ? 1 : 0;
      // the reference scans h0 below the bound for the copy
      ops++;
      r.bytes += 4ull * (unsigned long long)(len_h + h_v) + (LABELED ? (unsigned long long)len_h : 0ull);
    }
  }
  // PAIR_FRESH: path vertices whose adjacency to x has to be looked up
  int pv[4];
  const unsigned* prow[4];
  int known = 0, n_ask = 0;  // neighbours of every x, below the bound
  if (!LABELED && (kind == PAIR_FRESH || kind == PAIR_SHARED)) {
#pragma unroll
    for (int j = 0; j < 4; j++) { pv[j] = -1; prow[j] = nullptr; }
    for (int j = 0; j <= L; j++) {
      const int p = S.path[j];
      if (p >= ub_last) continue;
      if ((P.leaf_adj >> j) & 1u) known++;
      else {
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (k == n_ask) { pv[k] = p; prow[k] = hub_row(a, p); }
        n_ask++;
      }
    }
  }
  if constexpr (KIND == PAIR_SHARED) {
    // f(x) without v: x's degree less the path vertices next to it
    const int32_t* shared = S.ptr[P.parent[ms]];
    auto value = [&](int x, int& deg) {
      deg = (int)(a.rowptr[x + 1] - a.rowptr[x]);
      int f = deg - known;
      for (int i = 0; i < n_ask; i++) {
        const int p = i == 0 ? pv[0] : i == 1 ? pv[1] : i == 2 ? pv[2] : pv[3];
        const unsigned* row = i == 0 ? prow[0] : i == 1 ? prow[1] : i == 2 ? prow[2] : prow[3];
        const uint64_t pb = a.rowptr[p];
        f -= (row ? (__ldg(row + (x >> 5)) >> (x & 31)) & 1u
                  : bsearch_in<false>(a.colidx + pb, (int)(a.rowptr[p + 1] - pb), x)) ? 1 : 0;
      }
      return f;
    };
    unsigned long long sum_f = 0, sum_deg = 0;
    for (int i = lane; i < lenBm; i += 32) {
      int deg;
      sum_f += (unsigned)value(shared[i], deg);
      sum_deg += (unsigned)deg;
    }
    for (int d = 16; d; d >>= 1) {
      sum_f += __shfl_xor_sync(FULL, sum_f, d);
      sum_deg += __shfl_xor_sync(FULL, sum_deg, d);
    }
    if (mine) {
      const bool in_s = mode == MEMB_BITMAP ? leaf_member<MEMB_BITMAP>(set, v) : leaf_member<MEMB_FILTER>(set, v);
      unsigned long long f = sum_f, deg = sum_deg;
      if (in_s) {
        int dv;
        f -= (unsigned)value(v, dv);
        deg -= (unsigned)dv;
      }
      const unsigned long long k = (unsigned long long)(lenBm - (in_s ? 1 : 0));  // the main slot
      // members of s next to v, v aside: taken off below (each counts one, and
      // its bytes)
      int near = 0;
      const unsigned* row = hub_row(a, v);
      if (row && lenBm <= len) {
        for (int i = 0; i < lenBm; i++) {
          const int x = shared[i];
          near += x != v ? (__ldg(row + (x >> 5)) >> (x & 31)) & 1u : 0u;
        }
        len = 0;
      }
      f -= (unsigned)near;
      ops += k;
      r.cnt += f;
      r.bytes += 4ull * ((unsigned long long)lenBm + k) + 4ull * (deg + f);
    }
  }
  if (off) {  // the rest of a list whose operations are counted
    r = PairSums{0, 0, 0};
    ops = 0;
    rb += (unsigned)off;
    len -= mine ? off : 0;
    mine = false;
  }
  // walk
  constexpr int row_max = LABELED && KIND == PAIR_MEET ? kPairRow / 2 : kPairRow;
  int queued = 0;
  int total = len, next = e, next_off = 0, pair_take = 32;
  if (!PAGED) {
    int incl = min(len, 1 << 25);  // (the sum of 32 is an int; as long a list is taken by itself, in parts)
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += t;
    }
    total = __shfl_sync(FULL, incl, 31);
    if (total > row_max) {
      const int whole = __popc(__ballot_sync(FULL, incl <= row_max));  // candidates whose lists fit
      const int take = max(1, whole);
      if (lane >= take) {
        mine = false;
        r = PairSums{0, 0, 0};
        ops = 0;
      }
      if (lane >= whole) len = incl = 0;
      next = b + whole;
      next_off = whole ? 0 : off + row_max;
      pair_take = take;
      if (whole == 0 && lane == 0) len = row_max;
      total = __shfl_sync(FULL, whole ? incl : row_max, take - 1);
      incl = lane < whole ? incl : total;
    }
    S.prb[lane] = rb;
    S.pexcl[lane] = incl - len;
    if (lane == 31) S.pexcl[32] = total;
    __syncwarp();
  }
  if (lane == 0) {
    S.iter[L] = next;
    S.pair_off = next_off;
    S.pair_take = pair_take;
  }
  if (KIND != PAIR_SHARED) w.reads += __popc(__ballot_sync(FULL, mine));
  const int32_t* lists = LABELED ? a.colidx_lab : a.colidx;
  constexpr int U = 2;  // elements per lane in flight
  // (paged: one resolved list after the other)
  for (unsigned left = PAGED ? __ballot_sync(FULL, len > 0) : 1u; left; left &= left - 1) {
    const int one = PAGED ? __ffs(left) - 1 : 0;
    ListRef cur{nullptr, 0, -1};
    if (PAGED) {
      total = __shfl_sync(FULL, len, one);
      const unsigned long long base = __shfl_sync(FULL, rb, one);
      if (!gather_room(a, S, S.top[q], total, w)) break;
      cur = paged_list(a.pg, base, total, S.gather, S.pins, w.pc);
    }
    for (int t0 = 0; t0 < total; t0 += 32 * U) {
      int x[U], own[U];
      bool in[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        const int t = t0 + 32 * k + lane;
        in[k] = t < total;
        if (PAGED) {
          own[k] = one;
          x[k] = in[k] ? ld<PAGED>(cur.p + t, cur.cg) : 0;
        } else {
          int j = 0;
#pragma unroll
          for (int step = 16; step; step >>= 1)
            if (S.pexcl[j + step] <= t) j += step;
          own[k] = j;
          x[k] = in[k] ? __ldg(lists + S.prb[j] + (unsigned)(t - S.pexcl[j])) : 0;
        }
      }
      if (MET) {
        if (mode == MEMB_BITMAP) {
#pragma unroll
          for (int k = 0; k < U; k++) in[k] = in[k] && leaf_maybe<MEMB_BITMAP>(set, x[k]);
        } else {
#pragma unroll
          for (int k = 0; k < U; k++) in[k] = in[k] && leaf_maybe<MEMB_FILTER>(set, x[k]);
          if (__any_sync(FULL, any_of(in))) bsearch_n<false>(set.g, set.lenB, x, in, false);
        }
      } else if (!LABELED) {
        for (int i = 0; i <= L; i++) {
          const int p = S.path[i];
#pragma unroll
          for (int k = 0; k < U; k++) in[k] = in[k] && x[k] != p;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int vo = __shfl_sync(FULL, v, own[k]);
          in[k] = in[k] && x[k] != vo;
        }
      }
      if (MET && !__any_sync(FULL, any_of(in))) continue;
      int n_el = 0;
      if (KIND == PAIR_SHARED) {
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int vo = __shfl_sync(FULL, v, own[k]);
          n_el += in[k] && x[k] != vo ? 1 : 0;
        }
        r.cnt -= (unsigned)n_el;
        r.bytes -= 4ull * (unsigned)n_el;
        continue;
      }
#pragma unroll
      for (int k = 0; k < U; k++) n_el += in[k] ? 1 : 0;
      r.elems += (unsigned)n_el;
      if (KIND == PAIR_COPY) {
        bool hit[U];
        int h[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
          h[k] = __shfl_sync(FULL, h_v, own[k]);
          hit[k] = false;
          if (!LABELED) {
            const int vo = __shfl_sync(FULL, v, own[k]);
            hit[k] = in[k] && x[k] != vo;
          }
        }
        if (!LABELED) bsearch_n<false>(H0, len0, x, hit, false);
#pragma unroll
        for (int k = 0; k < U; k++) {
          if (!in[k]) continue;
          const int f = h[k] - (hit[k] ? 1 : 0);
          r.cnt += (unsigned)f;
          r.bytes += 4ull * (unsigned)(h[k] + f) + (LABELED ? (unsigned)h[k] : 0u);
        }
      } else if (KIND == PAIR_FRESH) {
        int deg[U], f[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
          deg[k] = f[k] = 0;
          if (!in[k]) continue;
          const uint64_t xb = a.rowptr[x[k]];
          deg[k] = (int)(a.rowptr[x[k] + 1] - xb);
          if (LABELED) {
            f[k] = label_range(a, x[k], last_group).y;
            if (a.T) f[k] = min(f[k], a.T);
          } else if (ub_last != INT_MAX) {
            deg[k] = lane_lower_bound(a.colidx + xb, deg[k], ub_last);
          }
        }
        if (!LABELED) {
#pragma unroll
          for (int k = 0; k < U; k++) f[k] = deg[k] - known - (__shfl_sync(FULL, v, own[k]) < ub_last ? 1 : 0);
          for (int i = 0; i < n_ask; i++) {
            const int p = i == 0 ? pv[0] : i == 1 ? pv[1] : i == 2 ? pv[2] : pv[3];
            const unsigned* row = i == 0 ? prow[0] : i == 1 ? prow[1] : i == 2 ? prow[2] : prow[3];
            bool hit[U];
#pragma unroll
            for (int k = 0; k < U; k++) hit[k] = in[k];
            if (row) {
#pragma unroll
              for (int k = 0; k < U; k++) hit[k] = in[k] && ((__ldg(row + (x[k] >> 5)) >> (x[k] & 31)) & 1u);
            } else {
              const uint64_t pb = a.rowptr[p];
              bsearch_n<false>(a.colidx + pb, (int)(a.rowptr[p + 1] - pb), x, hit, false);
            }
#pragma unroll
            for (int k = 0; k < U; k++) f[k] -= hit[k] ? 1 : 0;
          }
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          if (!in[k]) continue;
          r.cnt += (unsigned)f[k];
          r.bytes += 4ull * (unsigned)(deg[k] + f[k]) + (LABELED ? (unsigned)deg[k] : 0u);
        }
      } else {
        int4 en[U];
#pragma unroll
        for (int k = 0; k < U; k++)
          en[k] = in[k] ? *reinterpret_cast<const int4*>(S.memo + (x[k] & (a.memo_entries - 1))) : make_int4(-1, 0, 0, 0);
        int c = 0, by = 0, lw = 0;  // sums of these elements (an int holds them: kRowListMax)
        unsigned missing = 0;
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int h = __shfl_sync(FULL, h_v, own[k]), l1 = LABELED ? 0 : __shfl_sync(FULL, less, own[k]);
          const bool hit = in[k] && en[k].x == x[k] && (unsigned)en[k].y == epoch;
          if (in[k]) {
            c -= l1;
            by += h - l1;
          }
          if (hit) {
            c += en[k].z;
            by += en[k].w + en[k].z;
            lw += en[k].w;
          }
          missing |= in[k] && !hit ? 1u << k : 0u;
        }
        r.cnt += (unsigned long long)(long long)c;
        r.bytes += (unsigned long long)(4ll * by + (LABELED ? lw : 0));
        if (__any_sync(FULL, missing)) {
          for (int k = 0; k < U; k++) {
            const bool mk = (missing >> k) & 1u;
            const unsigned miss = __ballot_sync(FULL, mk);
            if (!miss) continue;
            int xk = x[0];
#pragma unroll
            for (int i = 1; i < U; i++) xk = k == i ? x[i] : xk;
            if (mk) S.queue[queued + __popc(miss & lanemask_lt())] = xk;
            queued += __popc(miss);
            __syncwarp();
            if (queued >= 32) {
              meet_values<LABELED>(a, S, set, mode, last_group, ub_last, 32, r);
              const int rest = lane < queued - 32 ? S.queue[32 + lane] : 0;
              __syncwarp();
              queued -= 32;
              if (lane < queued) S.queue[lane] = rest;
              __syncwarp();
            }
          }
        }
      }
    }
    if (PAGED) {
      __syncwarp();
      unpin(a.pg, cur);
    }
  }
  if (queued) meet_values<LABELED>(a, S, set, mode, last_group, ub_last, queued, r);
  // one operation per candidate and its copy, one per element; the main
  // operations' results are the elements
  unsigned long long cnt = r.cnt, bytes = r.bytes + 4ull * r.elems;
  ops += r.elems;
  for (int d = 16; d; d >>= 1) {
    cnt += __shfl_xor_sync(FULL, cnt, d);
    bytes += __shfl_xor_sync(FULL, bytes, d);
    ops += __shfl_xor_sync(FULL, ops, d);
  }
  w.setops += ops;
  w.bytes += bytes;
  return cnt;
}

// ---------------------------------------------------------------------
// Labeled plans that end in a chain -- single fresh levels from chain_from to
// the last: a path, a tail -- have a search below vertex path[chain_from] that
// depends on that vertex alone.  Its counts are worked out once per vertex of
// the right label, level by level from the end (chain_kernel, one launch per
// step for all plans of the launch), and the search adds the table's entry
// instead of descending.  A step reads each list part it needs once: bound by
// the gathers of the next level's entries.  Measured (B200), one launch, R-MAT
// graph of 65,536 vertices, 32 labels: the 7-path 13.6 -> 0.08 ms, the
// 5-cycle with a two-vertex tail 7.1 -> 4.7 ms.
// ---------------------------------------------------------------------
struct ChainStep {
  const ulonglong4* next;  // the level after's table (null: the last level, a length)
  ulonglong4* out;         // [n]: matches, set operations, algorithmic bytes, list reads below a vertex
  int32_t label;           // of the vertices the table is for
  int32_t part;            // label of the elements of their lists to add up
  int32_t leaf;            // next == null: label of the last level's list part
};
struct ChainSteps {
  ChainStep s[PM_MAX_BATCH];
};

__global__ void __launch_bounds__(256) chain_kernel(const __grid_constant__ ChainSteps steps, const uint64_t* rowptr,
                                                    const int32_t* colidx_lab, const int32_t* lab_off, int nl1,
                                                    const uint8_t* labels, int64_t n, int T) {
  const ChainStep& st = steps.s[blockIdx.y];
  const int lane = lane_id();
  auto range = [&](int64_t v, int l) {
    if (l >= nl1 - 1) return make_int2(0, 0);
    const int32_t* o = lab_off + v * nl1;
    return make_int2(o[l], o[l + 1] - o[l]);
  };
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long v0 = 32 * ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); v0 < n; v0 += 32 * warps) {
    unsigned todo = __ballot_sync(FULL, v0 + lane < n && labels[v0 + lane] == st.label);
    for (; todo; todo &= todo - 1) {
      const long long v = v0 + __ffs(todo) - 1;
      const uint64_t b = rowptr[v];
      const unsigned long long deg = rowptr[v + 1] - b;
      const int2 r = range(v, st.part);
      const int len = T ? min(r.y, T) : r.y;
      const int32_t* list = colidx_lab + b + r.x;
      unsigned long long cnt = 0, ops = 0, bytes = 0, reads = 0;
      for (int i0 = 0; i0 < len; i0 += 128) {
        int u[4];
#pragma unroll
        for (int q = 0; q < 4; q++) u[q] = i0 + 32 * q + lane < len ? list[i0 + 32 * q + lane] : -1;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (u[q] < 0) continue;
          if (st.next) {
            const ulonglong4 t = st.next[u[q]];
            cnt += t.x;
            ops += t.y;
            bytes += t.z;
            reads += t.w;
          } else {
            const unsigned long long du = rowptr[u[q] + 1] - rowptr[u[q]];
            const int k = range(u[q], st.leaf).y, kk = T ? min(k, T) : k;
            cnt += (unsigned long long)kk;
            ops++;
            bytes += 5ull * du + 4ull * (unsigned long long)kk;
          }
        }
      }
      for (int o = 16; o; o >>= 1) {
        cnt += __shfl_xor_sync(FULL, cnt, o);
        ops += __shfl_xor_sync(FULL, ops, o);
        bytes += __shfl_xor_sync(FULL, bytes, o);
        reads += __shfl_xor_sync(FULL, reads, o);
      }
      if (lane == 0)
        st.out[v] = make_ulonglong4(cnt, ops + 1, bytes + 5ull * deg + 4ull * (unsigned long long)len, reads + 1);
    }
  }
}

// Candidates [b, e) of the level before the chain: their entries added up.
__device__ __forceinline__ unsigned long long chain_sum(const DPlan& P, const int32_t* cand, int b, int e, Work& w) {
  unsigned long long cnt = 0, ops = 0, bytes = 0, reads = 0;
  for (int i = b + lane_id(); i < e; i += 32) {
    const ulonglong4 t = P.chain[cand[i]];
    cnt += t.x;
    ops += t.y;
    bytes += t.z;
    reads += t.w;
  }
  for (int o = 16; o; o >>= 1) {
    cnt += __shfl_xor_sync(FULL, cnt, o);
    ops += __shfl_xor_sync(FULL, ops, o);
    bytes += __shfl_xor_sync(FULL, bytes, o);
    reads += __shfl_xor_sync(FULL, reads, o);
  }
  w.setops += ops;
  w.bytes += bytes;
  w.reads += reads;
  return cnt;
}

template <bool LABELED, bool PAGED>
__device__ __forceinline__ unsigned long long pair_levels(const MatchArgs& a, const DPlan& P, WarpState& S, int L,
                                                          int b, int e, int off, Work* w) {
  const bool met = P.kind[P.level_begin[L + 1]] == SLOT_INTERSECT;
  if constexpr (!PAGED)
    if (P.pair == PAIR_MEET) return pair_pass<LABELED, PAGED, PAIR_MEET, false>(a, P, S, L, b, e, off, w);
  if constexpr (!LABELED && !PAGED)
    if (P.pair == PAIR_SHARED) return pair_pass<LABELED, PAGED, PAIR_SHARED, true>(a, P, S, L, b, e, off, w);
  if (P.pair == PAIR_COPY)
    return met ? pair_pass<LABELED, PAGED, PAIR_COPY, true>(a, P, S, L, b, e, off, w)
               : pair_pass<LABELED, PAGED, PAIR_COPY, false>(a, P, S, L, b, e, off, w);
  return met ? pair_pass<LABELED, PAGED, PAIR_FRESH, true>(a, P, S, L, b, e, off, w)
             : pair_pass<LABELED, PAGED, PAIR_FRESH, false>(a, P, S, L, b, e, off, w);
}

// A donated piece of a DFS: candidates [begin, end) of level `level`'s main
// slot under the path root(v0, v1), path[2..level].
struct Donation {
  int plan, root, level, begin, end;
  int path[7];  // path[2..level] used
  unsigned long long mul;  // the equal subtrees the piece stands for
};

// How often a busy warp looks for waiting warps (SM cycles, about 2 us).  A
// look costs one L2 read; a piece costs its taker the prefix again, so work
// that ends sooner than this is not worth handing out.
#define PM_CHECK_CYCLES 4096
constexpr unsigned kGroupSlots = 256;   // ring slots of a group
constexpr unsigned long long kQuit = ~0ull;         // a slot's mark: no more work
constexpr unsigned long long kClaimed = ~0ull - 1;  // a slot's mark: a piece is being written
constexpr unsigned kSchedStride = 16;   // words from one group's sched to the next (a line of its own)

__device__ __forceinline__ unsigned long long ld_vol_u64(const unsigned long long* p) {
  return *(const volatile unsigned long long*)p;
}

// Hands parts of the shallowest level range that is long enough to waiting
// warps.  sched counts tickets drawn by warps out of work and pieces handed
// out; their difference is the number of warps waiting, and a piece goes into
// the slot of the oldest unserved ticket, whose holder polls that slot alone
// -- so handing out is one CAS by the donor and no contention among the
// waiting (thousands of idle warps competing for one queue head by CAS cost
// several microseconds a piece and held every query with few roots at 5 us
// per donation).  A donor looks at its own group's word, then at another's,
// in turn: with one word for all warps 97% of the CAS failed (2.4 million on
// the labeled 5-cycle with a tail, launch 9.1 -> 4.5 ms).  With many waiting for each busy warp the range is cut into
// up to 33 pieces at once, one published per lane, so that a single heavy
// root reaches all warps in two or three rounds.  A range whose candidates
// head whole subtrees is long enough from 2 candidates on; one whose
// candidates only lead to the last level (one set operation each) needs
// `split` and is cut into pieces of at least half of that.
__device__ __noinline__ unsigned publish_pieces(const MatchArgs& a, const DPlan& P, WarpState& S, int L0, int L,
                                                int plan_id, int root_id) {
  const int n = P.nnodes;
  const int lane = lane_id();
  int k = L0, q = 0;
  unsigned g = 0;
  unsigned long long first = 0;
  if (lane == 0) {
    const unsigned own = blockIdx.x & (a.don_groups - 1);
    unsigned long long cur = 0;
    int waiting = 0;
    for (int look = 0; look < 2 && waiting <= 0; look++) {
      g = look == 0 ? own : (own + 1u + (unsigned)S.checks * 5u) & (a.don_groups - 1);
      cur = ld_vol_u64(a.sched + g * kSchedStride);
      waiting = (int)((unsigned)(cur >> 32) - (unsigned)cur);
    }
    if (waiting > 0) {
      const int busy = max(1, (int)(a.total_warps / a.don_groups) - waiting);
      const int want = min(32, (waiting + busy - 1) / busy);
      for (; k <= L; k++) {
        if ((P.copy_next >> k) & 1u) continue;  // one of its candidates is searched for all
        const int len = S.iend[k] - S.iter[k];
        // a candidate before a chain is one table entry: nothing to hand out;
        // those of a pass over the last two levels are lists, worth the prefix
        // their taker repeats in the number that a pass takes; where each warp
        // keeps values of its own (PAIR_MEET), in fewer than 32 they are worked
        // out again too often
        if (P.chain && k + 1 == P.chain_from) continue;
        const int unit = (k + 1 == n - 2) ? max(S.split, 2)
                         : !P.pair || k + 4 != n ? 2 : P.pair == PAIR_MEET ? 32 : max(2, S.pair_take);
        if (len < unit) continue;
        q = min(min(want, waiting), 2 * len / unit - 1);  // >= 1
        break;
      }
      if (q > 0) {
        // counted before they are given (draw_ticket must not see the takers
        // waiting still), taken back when another donor was first
        atomicAdd(a.all_sched, (unsigned long long)q);
        if (atomicCAS(a.sched + g * kSchedStride, cur, cur + (unsigned long long)q) != cur) {
          atomicAdd(a.all_sched, 0ull - (unsigned long long)q);
          q = 0;
        }
      }
      first = cur & 0xffffffffull;
    }
  }
  q = __shfl_sync(FULL, q, 0);
  if (q == 0) return 0;
  k = __shfl_sync(FULL, k, 0);
  g = __shfl_sync(FULL, g, 0);
  first = __shfl_sync(FULL, first, 0);
  const int it = S.iter[k], len = S.iend[k] - it;
  // part 0 of q + 1 stays here, part lane + 1 goes out
  const int b = it + (int)((long long)len * (lane + 1) / (q + 1));
  const int e = it + (int)((long long)len * (lane + 2) / (q + 1));
  const unsigned long long slot = first + (unsigned long long)lane;
  const unsigned at = g * kGroupSlots + (unsigned)(slot & (kGroupSlots - 1));
  // A slot is claimed before it is written: it may hold the piece of a ticket a
  // lap older or younger, which its taker is about to read, or another donor
  // may be writing one (a group with more warps than slots).  Each is gone when
  // its taker has read it: a bounded wait, in which no lane holds a claim.
  bool done = lane >= q;
  for (int spin = 0; spin < (1 << 20); spin++) {
    if (!done && atomicCAS(&a.don_ready[at], 0ull, kClaimed) == 0ull) {
      __threadfence();  // after the last taker's reads
      int4* dst = a.don_items + 3 * at;
      dst[0] = make_int4(plan_id, root_id, k, b);
      dst[1] = make_int4(e, S.path[2], S.path[3], S.path[4]);
      dst[2] = make_int4(S.path[5], S.path[6], (int)(unsigned)S.mul[k], (int)(unsigned)(S.mul[k] >> 32));
      st_release(&a.don_ready[at], slot + 1);
      done = true;
    }
    if (__all_sync(FULL, done)) break;
    __nanosleep(64);
  }
  __syncwarp();
  if (lane == 0) {
    S.iend[k] = it + len / (q + 1);
    atomicAdd(&a.stats[ST_SPLITS], (unsigned long long)q);
  }
  __syncwarp();
  return __all_sync(FULL, done) ? 0u : DEV_TIMEOUT;
}

// What was counted since (ops, bytes, reads) stands for m equal subtrees.
__device__ __forceinline__ void scale_work(Work& w, unsigned long long ops, unsigned long long bytes,
                                           unsigned long long reads, unsigned long long m) {
  w.setops = ops + (w.setops - ops) * m;
  w.bytes = bytes + (w.bytes - bytes) * m;
  w.reads = reads + (w.reads - reads) * m;
}

// Depth-first enumeration below a fixed path prefix.  path[0..L0] must be
// set; levels 1..L0 are computed here (for a donated piece this repeats the
// donor's work and is kept out of the counters), then candidates [b, e) of
// level L0's main slot (e < 0: all) are enumerated to the last level.
// Restates match() (src/gpu_match.cu:855-1047) without deferral: every
// branch is finished where it starts.
template <bool LABELED, bool PAGED>
__device__ unsigned long long dfs_from(const MatchArgs& a, const DPlan& P, WarpState& S, int L0, int b, int e,
                                       bool counted_prefix, int plan_id, int root_id, Work& w) {
  const int lane = lane_id();
  const int n = P.nnodes;
  if (lane == 0) S.top[1] = 0;
  __syncwarp();
  if (n == 3) {
    Work t;
    memset(&t, 0, sizeof(t));
    const unsigned long long c = (unsigned long long)count_slot<LABELED, PAGED>(a, P, S, 1, P.level_begin[1], 0, &t);
    add_work(w, t);
    return c;
  }
  if constexpr (LABELED && !PAGED) {
    if (P.chain && P.chain_from == 1) {  // a path: the root's second vertex says it all
      const ulonglong4 t = P.chain[S.path[1]];
      w.setops += t.y;
      w.bytes += t.z;
      w.reads += t.w;
      return t.x;
    }
  }
  const unsigned long long so = w.setops, by = w.bytes, rd = w.reads;
  unsigned long long cnt = 0;
  int L = 1;
  bool enter = true, prefix = true;  // level L's slots are still to be computed; L is on the given path
  while (true) {
    if (enter) {
      const long long c0 = clock64();
      const unsigned long long ops0 = w.setops, bytes0 = w.bytes, reads0 = w.reads;
      run_level<LABELED, PAGED>(a, P, S, L, w);
      if (LABELED && !prefix && P.copy_next) scale_work(w, ops0, bytes0, reads0, S.mul[L]);
      const unsigned long long cyc = (unsigned long long)(clock64() - c0);
      if (prefix && !counted_prefix) w.prefix_cyc += cyc;
      else w.level_cyc += cyc;
      if (w.err) return 0;
      if (L < L0) {
        L++;
        continue;
      }
      int it0 = 0, end0 = S.raw[P.level_begin[L]];
      if (prefix) {
        prefix = false;
        if (!counted_prefix) {
          w.setops = so;
          w.bytes = by;
          w.reads = rd;
        }
        it0 = b;
        if (e >= 0 && e < end0) end0 = e;
      }
      if (lane == 0) { S.iter[L] = it0; S.iend[L] = end0; }
      __syncwarp();
      enter = false;
    }
    // by the clock: the launch-wide deadline, the liveness signal for waiting
    // warps, and the look for waiting warps to hand work to (set operations
    // take from under a microsecond to hundreds, so counting them is no clock)
    if (__any_sync(FULL, clock64() >= S.next_check)) {
      int late = 0;
      if (lane == 0) {
        late = (global_ns() - S.t_start) > a.timeout_ns;
        late = late ? (int)DEV_TIMEOUT : 0;
        if ((S.checks++ & 15) == 0) {
          atomicAdd(a.heartbeat, 1ull);
          late |= (int)*(volatile unsigned int*)a.status;  // another warp failed: so has the launch
        }
      }
      late = __shfl_sync(FULL, late, 0);
      if (late) {
        w.err |= (unsigned)late;
        return 0;
      }
      bool worth = __any_sync(FULL, clock64() - S.began >= PM_CHECK_CYCLES);
      if constexpr (!LABELED && !PAGED)  // (a clique's matrix: long to build)
        worth = worth || (P.clique && a.clique_bits && S.size[P.level_begin[L] + 1] > 128);
      if (a.split_min > 0 && worth) {
        w.err |= publish_pieces(a, P, S, L0, L, plan_id, root_id);
        if (w.err) return 0;
      }
      if (lane == 0) S.next_check = clock64() + PM_CHECK_CYCLES;
      __syncwarp();
    }
    const int m = P.level_begin[L];
    const int it = S.iter[L];
    const int iend = S.iend[L];
    const unsigned long long ops0 = w.setops, bytes0 = w.bytes, reads0 = w.reads;
    // (labeled plans with levels of copies: what is searched here, for how many)
    const unsigned long long mul = LABELED && P.copy_next ? S.mul[L] : 1ull;
    bool subtree = false, bits = false;
    unsigned long long lanes_cnt = 0;
    if constexpr (!LABELED && !PAGED) {
      const int hs = P.level_begin[L] + 1;
      // (seven vertices: two levels between a candidate and the last make one
      // candidate of a large set too long a stretch without a look at the
      // deadline; the level below takes over there)
      bits = a.clique_bits && P.clique && L + 4 <= n && (L + 6 > n || S.size[hs] <= 128) && symmetric(a) && it < iend && S.size[hs] <= PM_CLIQUE_MAX &&
             S.top[L + 1] + clique_words(S.size[hs]) <= S.cap;
      subtree = !bits && P.l2_x >= 0 && L + 4 == n && it < iend && a.lane_subtree_max > 0 && (!a.T || distinct(a)) &&
                S.size[P.parent[P.l2_x]] <= a.lane_subtree_max &&
                S.top[L + 1] + 32ll * S.size[P.parent[P.l2_x]] <= S.cap;
    }
    bool chain = false;
    if constexpr (LABELED && !PAGED) {
      chain = P.chain && L + 1 == P.chain_from && it < iend;
      if (chain) {
        const long long c0 = clock64();
        const int e2 = min(iend, it + 2048);
        cnt += mul * chain_sum(P, S.ptr[m], it, e2, w);
        if (P.copy_next) scale_work(w, ops0, bytes0, reads0, mul);
        w.leaf_cyc += (unsigned long long)(clock64() - c0);
        if (lane == 0) S.iter[L] = e2;
        __syncwarp();
      }
    }
    if (chain) {
      // done above
    } else if (!bits && it < iend && L + 4 == n && pair_ready<LABELED, PAGED>(a, P, S)) {
      const int off = S.pair_off;
      const int e2 = off ? it + 1 : min(iend, it + 32);
      const long long c0 = clock64();
      Work t;
      memset(&t, 0, sizeof(t));
      cnt += mul * pair_levels<LABELED, PAGED>(a, P, S, L, it, e2, off, &t);
      add_work(w, t);
      if (LABELED && P.copy_next) scale_work(w, ops0, bytes0, reads0, mul);
      w.leaf_cyc += (unsigned long long)(clock64() - c0);
      __syncwarp();  // (where to go on: pair_pass wrote it)
      if (w.err) return 0;
    } else if (bits) {
      // (a look for waiting warps between: every candidate below a large set
      // may be long, the more so with levels between it and the last)
      const int e2 = min(iend, it + (S.size[P.level_begin[L] + 1] <= 32 ? 32 : L + 4 == n ? 8 : 1));
      const long long c0 = clock64();
      unsigned long long ops, bytes, reads;
      cnt += clique_bits(a, P, S, L, it, e2, &ops, &bytes, &reads);
      w.setops += ops;
      w.bytes += bytes;
      w.reads += reads;
      w.leaf_cyc += (unsigned long long)(clock64() - c0);
      if (lane == 0) S.iter[L] = e2;
      __syncwarp();
    } else if (subtree && lane_subtree(a, P, S, L, it, min(iend, it + 32), w, &lanes_cnt)) {
      cnt += lanes_cnt;
      if (lane == 0) S.iter[L] = min(iend, it + 32);
      __syncwarp();
    } else if (it < iend && L + 1 == n - 2) {
      const int e2 = min(iend, it + PM_LEAF_BATCH);
      const long long c0 = clock64();
      cnt += mul * leaf_batch<LABELED, PAGED>(a, P, S, L, it, e2, w);
      if (LABELED && P.copy_next) scale_work(w, ops0, bytes0, reads0, mul);
      w.leaf_cyc += (unsigned long long)(clock64() - c0);
      if (lane == 0) S.iter[L] = e2;
      __syncwarp();
      if (w.err) return 0;
    } else if (it < iend) {
      const int v = S.ptr[m][it];
      const bool skip = !LABELED && S.raw[m] != S.size[m] && on_path(S, L, v);
      // a level of copies does not read v: one candidate is searched for all
      const bool same = LABELED && ((P.copy_next >> L) & 1u);
      __syncwarp();
      if (lane == 0) {
        S.iter[L] = same ? iend : it + 1;
        S.path[L + 1] = v;
        S.mul[L + 1] = same ? mul * (unsigned long long)(iend - it) : mul;
      }
      __syncwarp();
      if (skip) continue;
      L++;
      enter = true;
    } else {
      L--;
      if (L < L0) break;
    }
  }
  return cnt;
}

// Draws a ticket: the warp is out of work and will take the piece that lands
// in the ticket's slot.  The warp whose ticket leaves none of the started
// warps busy (pieces are counted before they are published, so their takers
// count as busy) marks every slot a warp can be waiting on with kQuit.  Warps
// that have not started hold nothing: the root queue is empty by now, and
// they will find their own ticket's slot marked -- so the end does not wait
// for blocks that other launches keep from starting.  A warp counts itself
// started before its first pop, and the count is read here after a pop that
// found the queue empty, so no warp with roots is missed.  `seen` is the
// largest count this warp has read: it only grows, so fewer waiting warps
// than that need no new look.  Returns the ticket, or kQuit for the last warp.
__device__ unsigned long long draw_ticket(const MatchArgs& a, unsigned& seen) {
  const int lane = lane_id();
  unsigned long long old = 0;
  unsigned ticket = 0;
  __syncwarp();
  if (lane == 0) {
    ticket = (unsigned)(atomicAdd(a.sched + (blockIdx.x & (a.don_groups - 1)) * kSchedStride, 1ull << 32) >> 32);
    old = atomicAdd(a.all_sched, 1ull << 32);
  }
  ticket = __shfl_sync(FULL, ticket, 0);
  old = __shfl_sync(FULL, old, 0);
  const int waiting = (int)((unsigned)(old >> 32) + 1u - (unsigned)old);
  if (waiting < (int)seen) return ticket;
  if (lane == 0) {
    __threadfence();  // after the pop that found the queue empty
    seen = atomicAdd(a.started, 0u);
  }
  seen = __shfl_sync(FULL, seen, 0);
  if (waiting != (int)seen) return ticket;
  for (unsigned i = lane; i < a.don_groups * kGroupSlots; i += 32)
    *(volatile unsigned long long*)&a.don_ready[i] = kQuit;
  return kQuit;
}

// One look at the ticket's slot: 0 nothing yet, 1 a piece (in d), -1 no more
// work.
__device__ int wait_piece(const MatchArgs& a, unsigned long long ticket, Donation& d) {
  int got = 0;
  int v[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (lane_id() == 0) {
    const unsigned at =
        (blockIdx.x & (a.don_groups - 1)) * kGroupSlots + (unsigned)(ticket & (kGroupSlots - 1));
    unsigned long long* ready = &a.don_ready[at];
    // polled with plain volatile reads: an acquire read drops the SM's L1
    // contents, which the busy warps beside this one live on
    const unsigned long long r = ld_vol_u64(ready);
    if (r == kQuit) got = -1;
    else if (r == ticket + 1 && ld_acquire(ready) == r) {
      got = 1;
      const volatile int* src = (const volatile int*)(a.don_items + 3 * at);
      for (int i = 0; i < 12; i++) v[i] = src[i];
      st_release(ready, 0ull);  // read: the slot is free for the ticket one lap on
    }
  }
  got = __shfl_sync(FULL, got, 0);
  if (got <= 0) return got;
  int u[12];
#pragma unroll
  for (int i = 0; i < 12; i++) u[i] = __shfl_sync(FULL, v[i], 0);
  d.plan = u[0];
  d.root = u[1];
  d.level = u[2];
  d.begin = u[3];
  d.end = u[4];
  d.path[0] = 0;
  d.path[1] = 0;
  d.path[2] = u[5];
  d.path[3] = u[6];
  d.path[4] = u[7];
  d.path[5] = u[8];
  d.path[6] = u[9];
  d.mul = (unsigned long long)(unsigned)u[11] << 32 | (unsigned)u[10];
  return 1;
}

// MINB = 4: 64 registers, four 256-thread blocks per SM (more warps in flight,
// some spills); MINB = 3: 85 registers, three blocks; MINB = 1: up to 128
// registers, no spills, fewer warps.
template <bool LABELED, bool PAGED, int MINB>
__global__ void __launch_bounds__(MINB == 1 ? 512 : 256, MINB) match_kernel(const __grid_constant__ MatchArgs a) {
  extern __shared__ WarpState smem_state[];
  // What the block's warps have in common: thousands of warps adding their
  // counters to the same few words, one atomic after the other, took longer
  // than a small query's search (the 4-clique on 400 vertices: launch 57 ->
  // 48 us).
  __shared__ unsigned long long blk_stats[kStatWords];
  __shared__ unsigned blk_empty, blk_ended;  // plans whose queue was found empty; warps that have ended
  if (threadIdx.x < kStatWords) blk_stats[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    blk_empty = blk_ended = 0;
    atomicAdd(a.started, blockDim.x >> 5);  // before the first pop (draw_ticket)
    __threadfence();
  }
  __syncthreads();
  const int lane = lane_id();
  const int wib = threadIdx.x >> 5;
  WarpState& S = smem_state[wib];
  const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + wib;
  int32_t* own = a.arena + gw * a.arena_words;
  if (lane == 0) {
    S.next_check = 0;
    S.checks = 0;
    S.next_id = 0;
    S.sb_id = 0;
    S.cq_id = 0;
    S.memo = a.memo ? a.memo + gw * (a.memo_entries + 1) : nullptr;
    S.memo_epoch = a.memo ? (uint32_t)S.memo[a.memo_entries].x : 0u;
    S.memo_id = 0;
    S.memo_len = -1;
    S.memo_ub = 0;
    S.pair_take = 32;
    S.pair_off = 0;
    for (int k = 0; k < 16; k++) S.ptr[k] = nullptr;
    S.t_start = global_ns();
    S.arena = own;
    S.cap = a.slot_words;
    S.gather = own + a.slot_words;
    S.ghalf = (int32_t)(a.gather_words / 2);
    S.big = -1;
    S.mphase = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  Work w;
  memset(&w, 0, sizeof(w));
  unsigned long long roots = 0;
  const int np = a.nplans;
  int p = 0;
  int exhausted = 0;
  long long r = 0, re = 0;        // phase 1: roots [r, re) of the last pop
  unsigned long long local = 0;   // matches of plan `plan` not yet in a.counts
  int plan = p;
  // phase 2: the ticket, and for how long
  bool waiting = false;
  unsigned long long ticket = kQuit, last_beat = 0, last_change = 0, t_drain = 0, busy_ns = 0, t_item = 0;
  unsigned seen = 0;
  int looks = 0;
  while (!w.err) {
    Donation item;
    item.level = 1;
    item.begin = 0;
    item.end = -1;
    item.mul = 1;
    bool whole = true;  // a root, not a piece of one
    if (r < re) {
      // position r of the range; with an order, the order's entry there
      const long long pos = a.plans[plan].rbase + r;
      item.root = (int)(a.root_order ? (long long)a.root_order[pos] : pos);
      r++;
      roots++;
    } else if (exhausted < np) {
      // phase 1: root chunks from the per-plan cursors, one plan after the
      // other: warps on twenty plans at once empty each other's instruction
      // cache and their own value tables (20 patterns on 65,536 vertices, each
      // warp starting on another plan 21.4 ms, so 19.2 ms)
      if (lane == 0 && local) atomicAdd(&a.counts[plan], local);
      local = 0;
      const DPlan& P = a.plans[p];
      // a pop is `pop` roots of one shard unit of `chunk` roots (the last pop of
      // a unit, and the last unit, may be shorter)
      const unsigned long long per = (unsigned long long)((a.chunk + a.pop - 1) / a.pop);
      const unsigned long long nchunks = (unsigned long long)((P.nroots + a.chunk - 1) / a.chunk);
      unsigned long long c = ~0ull;
      if (lane == 0 && !((*(volatile unsigned*)&blk_empty >> p) & 1u)) c = atomicAdd(&a.cursors[p], 1ull);
      c = __shfl_sync(FULL, c, 0);
      if (c == ~0ull) {
        p = (p + 1 == np) ? 0 : p + 1;
        exhausted++;
        continue;
      }
      const unsigned long long gc = c / per * (unsigned long long)a.shard_count + (unsigned long long)a.shard_rank;
      plan = p;
      if (gc >= nchunks) {
        if (lane == 0) atomicOr(&blk_empty, 1u << plan);
        p = (p + 1 == np) ? 0 : p + 1;
        exhausted++;
        continue;
      }
      const long long sub = (long long)(c % per) * a.pop;  // within the unit
      exhausted = 0;
      if (PAGED && a.pf_off && plan == 0 && sub == 0) {
        // post the predicted pages of a chunk this warp's successors will reach
        const long long pc = (long long)gc + (long long)a.pf_ahead * a.shard_count;
        // only while the host's queue is short: a page posted behind a long
        // queue stays LOADING, and warps that miss on it meanwhile can neither
        // read it from a frame nor load it themselves
        unsigned long long queued = 0;
        if (lane == 0)
          queued = *(volatile unsigned long long*)a.pg.ring_head - *(volatile unsigned long long*)a.pg.host_tail;
        queued = __shfl_sync(FULL, queued, 0);  // one decision for the warp (the block below shuffles)
        if (pc < a.pf_chunks && queued < 64) {
          PageCounters lpc = {};
          for (int k = a.pf_off[pc] + lane; k < a.pf_off[pc + 1]; k += 32) {
            const int32_t pg = a.pf_pages[k];
            if (pg >= 0 && pg < a.pg.n_pages && ld_vol(&a.pg.page_frame[pg]) == PAGE_ABSENT)
              request_page(a.pg, pg, lpc);
          }
          unsigned long long v[3] = {lpc.requests, lpc.evictions, lpc.dropped};
#pragma unroll
          for (int q = 0; q < 3; q++)
            for (int o = 16; o; o >>= 1) v[q] += __shfl_xor_sync(FULL, v[q], o);
          w.pc.requests += v[0];
          w.pc.evictions += v[1];
          w.pc.dropped += v[2];
          w.prefetched += v[0];
        }
      }
      r = (long long)gc * a.chunk + sub;
      re = min((long long)P.nroots, (long long)gc * a.chunk + min((long long)a.chunk, sub + a.pop));
      continue;
    } else {
      // phase 2: take pieces until every warp is out of work
      if (!waiting) {
        if (lane == 0 && local) atomicAdd(&a.counts[plan], local);
        local = 0;
        last_change = global_ns();
        if (!t_drain) t_drain = last_change;
        if (t_item) busy_ns += last_change - t_item;
        ticket = draw_ticket(a, seen);
        if (ticket == kQuit) break;
        waiting = true;
        looks = 0;
      }
      const int got = wait_piece(a, ticket, item);
      if (got < 0) break;
      if (got == 0) {
        // poll the one word; the clock, the heartbeat and the status (words
        // all waiting warps share) only every 64th time
        __nanosleep(looks < 64 ? 100 : 400);
        if (++looks & 63) continue;
        unsigned long long beat = 0;
        unsigned int failed = 0;
        if (lane == 0) {
          beat = ld_vol_u64(a.heartbeat);
          failed = *(volatile unsigned int*)a.status;
        }
        beat = __shfl_sync(FULL, beat, 0);
        if (__shfl_sync(FULL, failed, 0)) break;
        // bounded wait: give up (and report DEV_TIMEOUT) when no warp has made
        // progress for timeout_ns
        const unsigned long long now = global_ns();
        if (beat != last_beat) { last_beat = beat; last_change = now; }
        else if (__any_sync(FULL, now > last_change && now - last_change > a.timeout_ns)) {
          if (lane == 0) atomicOr(a.status, (unsigned)DEV_TIMEOUT);
          break;
        }
        continue;
      }
      waiting = false;
      whole = false;
      plan = item.plan;
      t_item = global_ns();
    }
    const DPlan& P = a.plans[plan];
    const int2 e = P.roots[item.root];
    if (lane == 0) {
      S.path[0] = e.x;
      S.path[1] = e.y;
      S.mul[item.level] = item.mul;
      for (int k = 2; k <= item.level; k++) S.path[k] = item.path[k];
      S.split = (a.root_split && plan == 0) ? a.root_split[item.root] : a.split_min;
      S.began = clock64();
    }
    __syncwarp();
    const unsigned long long b0 = w.bytes, r0 = w.reads;
    const unsigned long long c0 = dfs_from<LABELED, PAGED>(a, P, S, item.level, item.begin, item.end, whole, plan,
                                                           item.root, w);
    return_arena(a, S, own);
    local += c0;
    if (lane == 0 && plan == 0) {
      if (a.root_counts) atomicAdd(&a.root_counts[item.root], c0);
      if (a.root_cost) atomicAdd(&a.root_cost[item.root], (float)(w.bytes - b0 + (whole ? 8 : 0)));
      if (a.root_reads) atomicAdd(&a.root_reads[item.root], (float)(w.reads - r0));
    }
  }
  // a warp that failed draws no ticket (a piece given to it would be lost):
  // the status word ends the others' wait
  if (w.err && lane == 0) atomicOr(a.status, w.err);
  __syncwarp();
  if (lane == 0) {
    if (a.memo) S.memo[a.memo_entries].x = (int32_t)S.memo_epoch;
    const unsigned long long t_end = global_ns();
    auto add = [&](int k, unsigned long long v) {
      if (v) atomicAdd(&blk_stats[k], v);
    };
    add(ST_WARP_NS, t_end - S.t_start);
    if (t_drain) add(ST_IDLE_NS, t_end - t_drain - min(busy_ns, t_end - t_drain));
    add(ST_SETOPS, w.setops);
    add(ST_BYTES, w.bytes + 8ull * roots);
    add(ST_ROOTS, roots);
    add(ST_BORROWS, w.borrows);
    add(ST_LEAF_CYC, w.leaf_cyc);
    add(ST_LEVEL_CYC, w.level_cyc);
    add(ST_PREFIX_CYC, w.prefix_cyc);
    add(ST_PREFETCH, w.prefetched);
    if (PAGED) {
      add(ST_HITS, w.pc.hits);
      add(ST_MISSES, w.pc.misses);
      add(ST_ZC_BYTES, w.pc.zc_bytes);
      add(ST_REQUESTS, w.pc.requests);
      add(ST_EVICTIONS, w.pc.evictions);
      add(ST_DROPPED, w.pc.dropped);
      add(ST_DEV_LOADS, w.pc.dev_loads);
      add(ST_DEV_BYTES, w.pc.dev_bytes);
    }
    // the block's last warp takes the sums out
    __threadfence_block();
    if (atomicAdd(&blk_ended, 1u) == (blockDim.x >> 5) - 1) {
      __threadfence_block();
      for (int k = 0; k < kStatWords; k++) {
        const unsigned long long v = *(volatile unsigned long long*)&blk_stats[k];
        if (v) atomicAdd(&a.stats[k], v);
      }
    }
  }
}

// =====================================================================
// Root filter (restates JobQueuePreprocessor, src/job_queue.h:39-64, as
// three passes: per-vertex max neighbour degree, per-vertex root counts +
// scan, ordered write).  Root order = reference order (r ascending, then
// adjacency order), so root ids match the reference's Job[] indices.
// =====================================================================

// Also sums a hash of every entry's vertex pair into asym[0], with the sign of
// the entry's direction: 0 when each entry has its reverse (and, but for one
// graph in 2^64 or so, only then).  asym[1]: bit 0 a list holds an element
// twice, bit 1 a list holds its own vertex.
__device__ __forceinline__ unsigned long long pair_hash(unsigned lo, unsigned hi) {
  uint64_t x = ((uint64_t)hi << 32 | lo) + 0x9E3779B97F4A7C15ull;
  return Rng::splitmix(x);
}

__global__ void __launch_bounds__(512) maxnbrdeg_kernel(const uint64_t* rowptr, const int32_t* colidx, int64_t n,
                                                        int32_t* out, unsigned long long* asym) {
  __shared__ int best[kListWarps];
  const int lane = lane_id();
  unsigned long long sum = 0;
  bool twice = false, loop = false;
  auto walk = [&](long long v, uint64_t b, uint64_t e, uint64_t e_list) {
    int m = 0;
    for (uint64_t i0 = b; i0 < e; i0 += 128) {
      int u[4];
#pragma unroll
      for (int q = 0; q < 4; q++) u[q] = i0 + 32 * q + lane < e ? colidx[i0 + 32 * q + lane] : -1;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (u[q] < 0) continue;
        const uint64_t next = i0 + 32 * q + lane + 1;
        twice = twice || (next < e_list && colidx[next] == u[q]);
        m = max(m, (int)(rowptr[u[q] + 1] - rowptr[u[q]]));
        if (u[q] > v) sum += pair_hash((unsigned)v, (unsigned)u[q]);
        else if (u[q] < v) sum -= pair_hash((unsigned)u[q], (unsigned)v);
        else loop = true;
      }
    }
    return __reduce_max_sync(FULL, m);
  };
  for_lists(rowptr, 0, n,
            [&](long long v, uint64_t b, uint64_t e) {
              const int m = walk(v, b, e, e);
              if (lane == 0) out[v] = m;
            },
            [&](long long v, uint64_t, uint64_t e, uint64_t b0, uint64_t e0, int k) {
              const int m = walk(v, b0, e0, e);
              if (lane == 0) best[k] = m;
              __syncthreads();
              if (threadIdx.x < 32) {
                const int top = __reduce_max_sync(FULL, lane < kListWarps ? best[lane] : 0);
                if (lane == 0) out[v] = top;
              }
              __syncthreads();
            });
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
  if (lane == 0 && sum) atomicAdd(asym, sum);
  const unsigned odd = (__any_sync(FULL, twice) ? 1u : 0u) | (__any_sync(FULL, loop) ? 2u : 0u);
  if (odd && lane == 0) atomicOr(asym + 1, (unsigned long long)odd);
}

// Regroups each list by label, keeping id order within a label (a stable
// partition), ranks from __match_any_sync; a long list's warps count the
// labels of their parts first.  Vertices [v_begin, v_end); entry i of the
// adjacency array lands at out[i - out_base].
__global__ void __launch_bounds__(512) label_group_kernel(const uint64_t* rowptr, const int32_t* colidx,
                                                          const uint8_t* labels, int64_t v_begin, int64_t v_end,
                                                          int nl1, int32_t* out, uint64_t out_base, int32_t* off) {
  __shared__ int base_s[kListWarps][33];
  const int lane = lane_id();
  const int wib = threadIdx.x >> 5;
  int* base = base_s[wib];
  // entries of each label in [b, e) into base[]
  auto count = [&](uint64_t b, uint64_t e) {
    base[lane] = 0;
    __syncwarp();
    for (uint64_t i0 = b; i0 < e; i0 += 128) {
      int x[4], lb[4];
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = i0 + 32 * q + lane < e ? colidx[i0 + 32 * q + lane] : -1;
#pragma unroll
      for (int q = 0; q < 4; q++) lb[q] = x[q] >= 0 ? (int)labels[x[q]] : -1;
#pragma unroll
      for (int q = 0; q < 4; q++)
        if ((unsigned)lb[q] < 32u) atomicAdd(&base[lb[q]], 1);
    }
    __syncwarp();
  };
  auto scan = [&](int mine) {  // exclusive sum over the lanes
    int incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    return incl - mine;
  };
  // entries [b, e) to their places, base[] the next place of each label in the list at b_list
  auto place = [&](uint64_t b_list, uint64_t b, uint64_t e) {
    for (uint64_t i0 = b; i0 < e; i0 += 128) {
      int x[4], lb[4];
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = i0 + 32 * q + lane < e ? colidx[i0 + 32 * q + lane] : -1;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        lb[q] = x[q] >= 0 ? (int)labels[x[q]] : 32 + lane;  // none: matches only itself
        if (lb[q] >= 32) x[q] = -1;                         // (no such label is accepted)
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const unsigned same = __match_any_sync(FULL, lb[q]);
        if (x[q] >= 0) out[b_list - out_base + base[lb[q]] + __popc(same & lanemask_lt())] = x[q];
        __syncwarp();
        if (x[q] >= 0 && (same & lanemask_lt()) == 0) base[lb[q]] += __popc(same);
        __syncwarp();
      }
    }
  };
  auto offsets = [&](long long v, uint64_t b, uint64_t e, int excl) {
    if (lane < nl1 - 1) off[v * nl1 + lane] = excl;
    if (lane == 0) off[v * nl1 + nl1 - 1] = (int)(e - b);  // up to 32 labels: entry 32 needs its own store
  };
  for_lists(rowptr, v_begin, v_end,
            [&](long long v, uint64_t b, uint64_t e) {
              count(b, e);
              const int excl = scan(base[lane]);
              offsets(v, b, e, excl);
              __syncwarp();
              base[lane] = excl;
              __syncwarp();
              place(b, b, e);
            },
            [&](long long v, uint64_t b, uint64_t e, uint64_t b0, uint64_t e0, int k) {
              count(b0, e0);
              __syncthreads();
              if (wib == 0) {  // lane l: label l's entries in the parts before each part
                int mine = 0;
                for (int w = 0; w < kListWarps; w++) {
                  const int c = base_s[w][lane];
                  base_s[w][lane] = mine;
                  mine += c;
                }
                const int excl = scan(mine);
                offsets(v, b, e, excl);
                for (int w = 0; w < kListWarps; w++) base_s[w][lane] += excl;
              }
              __syncthreads();
              place(b, b0, e0);
              __syncthreads();
            });
}

// Vertices per power of two of their degree (bin k: degree in [2^k, 2^(k+1))).
__global__ void degree_bins_kernel(const uint64_t* rowptr, int64_t n, unsigned int* bins) {
  __shared__ unsigned int b[32];
  if (threadIdx.x < 32) b[threadIdx.x] = 0;
  __syncthreads();
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const unsigned deg = (unsigned)(rowptr[v + 1] - rowptr[v]);
    if (deg) atomicAdd(&b[31 - __clz(deg)], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 32 && b[threadIdx.x]) atomicAdd(&bins[threadIdx.x], b[threadIdx.x]);
}

// Gives every vertex of at least min_deg neighbours a bit row and fills it
// (rows zeroed before).
__global__ void __launch_bounds__(512) hub_rows_kernel(const uint64_t* rowptr, const int32_t* colidx, int64_t n,
                                                       int min_deg, int64_t words, unsigned int* next, int32_t* slot,
                                                       unsigned int* bits) {
  __shared__ int row;
  const int lane = lane_id();
  auto fill = [&](int k, uint64_t b, uint64_t e) {
    for (uint64_t i = b + lane; i < e; i += 32) {
      const int u = colidx[i];
      if (u >= 0 && u < n) atomicOr(&bits[k * words + (u >> 5)], 1u << (u & 31));
    }
  };
  for_lists(rowptr, 0, n,
            [&](long long v, uint64_t b, uint64_t e) {
              int k = -1;
              if ((long long)(e - b) >= min_deg) {
                if (lane == 0) k = (int)atomicAdd(next, 1u);
                k = __shfl_sync(FULL, k, 0);
                fill(k, b, e);
              }
              if (lane == 0) slot[v] = k;
            },
            [&](long long v, uint64_t b, uint64_t e, uint64_t b0, uint64_t e0, int) {
              const bool has = (long long)(e - b) >= min_deg;
              if (threadIdx.x == 0) {
                row = has ? (int)atomicAdd(next, 1u) : -1;
                slot[v] = row;
              }
              __syncthreads();
              if (has) fill(row, b0, e0);
              __syncthreads();
            });
}

struct RootFilter {
  int labeled;
  int need_gt;   // unlabeled with partial[0]==1: keep r > c only
  int lab0, lab1;
  int d0, d1, d2;
};

template <bool WRITE>
__global__ void __launch_bounds__(512) roots_kernel(const uint64_t* rowptr, const int32_t* colidx,
                                                    const uint8_t* labels, const int32_t* maxnbrdeg, int64_t n,
                                                    RootFilter f, int32_t* counts, const int64_t* offsets, int2* out) {
  __shared__ int part_total[kListWarps];
  const int lane = lane_id();
  // root edges (r, c) for c in [b, e): counted, or written from out[base] on
  auto filter = [&](long long r, uint64_t b, uint64_t e, bool write, long long base) {
    int total = 0;
    for (uint64_t i0 = b; i0 < e; i0 += 128) {
      int c[4];
      bool keep[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        c[q] = i0 + 32 * q + lane < e ? colidx[i0 + 32 * q + lane] : -1;
        keep[q] = c[q] >= 0 && (!f.need_gt || r > c[q]);
      }
      if (f.labeled) {
#pragma unroll
        for (int q = 0; q < 4; q++) keep[q] = keep[q] && labels[c[q]] == f.lab1;
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
        keep[q] = keep[q] && (int)(rowptr[c[q] + 1] - rowptr[c[q]]) >= f.d1 && maxnbrdeg[c[q]] >= f.d2;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const unsigned bal = __ballot_sync(FULL, keep[q]);
        if (write && keep[q]) out[base + total + __popc(bal & lanemask_lt())] = make_int2((int)r, c[q]);
        total += __popc(bal);
      }
    }
    return total;
  };
  auto root_ok = [&](long long r, uint64_t b, uint64_t e) {
    return (long long)(e - b) >= f.d0 && (!f.labeled || labels[r] == f.lab0);
  };
  for_lists(rowptr, 0, n,
            [&](long long r, uint64_t b, uint64_t e) {
              const int total = root_ok(r, b, e) ? filter(r, b, e, WRITE, WRITE ? offsets[r] : 0) : 0;
              if (!WRITE && lane == 0) counts[r] = total;
            },
            [&](long long r, uint64_t b, uint64_t e, uint64_t b0, uint64_t e0, int k) {
              if (!root_ok(r, b, e)) {
                if (!WRITE && threadIdx.x == 0) counts[r] = 0;
                return;  // the same for all of the block
              }
              const int mine = filter(r, b0, e0, false, 0);
              if (lane == 0) part_total[k] = mine;
              __syncthreads();
              int before = 0, all = 0;
              for (int w = 0; w < kListWarps; w++) {
                if (w < k) before += part_total[w];
                all += part_total[w];
              }
              if (WRITE) filter(r, b0, e0, true, offsets[r] + before);
              else if (threadIdx.x == 0) counts[r] = all;
              __syncthreads();
            });
}

// =====================================================================
// Host glue
// =====================================================================

namespace {

void free_dev(void* p) { if (p) cudaFree(p); }

pm_status ensure(void** p, size_t* have, size_t want) {
  if (*have >= want && *p) return PM_OK;
  free_dev(*p);
  *p = nullptr;
  *have = 0;
  if (want == 0) return PM_OK;
  cudaError_t e = cudaMalloc(p, want);
  if (e != cudaSuccess) {
    *p = nullptr;
    return fail(PM_ERR_OOM, "cudaMalloc(%zu) failed: %s", want, cudaGetErrorString(e));
  }
  *have = want;
  return PM_OK;
}

pm_status check_device(int device) {
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0)
    return fail(PM_ERR_NO_DEVICE, "no CUDA device available (%s); libpumatch_b200 has no CPU path",
                e == cudaSuccess ? "0 devices" : cudaGetErrorString(e));
  if (device < 0 || device >= count) return fail(PM_ERR_INVALID, "device %d out of range", device);
  CK(cudaSetDevice(device));
  return PM_OK;
}

DPlan to_dplan(const Plan& p) {
  DPlan d;
  memset(&d, 0, sizeof(d));
  d.nnodes = p.nnodes;
  d.nslots = p.nslots;
  d.labeled = p.labeled;
  d.last_slot = p.level_begin[p.nnodes - 2];
  for (int i = 0; i <= PM_MAX_PAT; i++) d.level_begin[i] = p.level_begin[i];
  for (int s = 0; s < 16; s++) d.alias[s] = -1;
  for (int s = 0; s < p.nslots; s++) {
    d.slot_labels[s] = p.slot_labels[s];
    d.partial[s] = p.partial[s];
    d.kind[s] = (uint8_t)slot_kind(p.set_ops[s]);
    d.parent[s] = (uint8_t)slot_parent(p.set_ops[s]);
  }
  // Slots of one level with the same operation, operands, labels and partial
  // order differ only in how their bound combines the constrained path
  // vertices: the main slot takes the smallest, helpers the largest.  A
  // helper equal to an earlier helper is that helper; the main slot is the
  // prefix of such a helper below its own (smaller) bound -- also under
  // truncation, since both keep their first survivors in the same order.
  for (int L = 1; L + 2 < p.nnodes; L++) {
    const int b = p.level_begin[L], e = p.level_begin[L + 1];
    for (int i = b + 1; i <= e; i++) {
      const int s = (i == e) ? b : i;  // helpers first, the main slot last
      for (int t = b + 1; t < e; t++) {
        if (t == s || (s != b && t >= s)) continue;
        if (p.set_ops[s] != p.set_ops[t] || p.slot_labels[s] != p.slot_labels[t] || p.partial[s] != p.partial[t])
          continue;
        if (d.alias[t] >= 0) continue;  // alias a computed slot only
        d.alias[s] = (int8_t)t;
        d.alias_prefix[s] = (s == b) ? 1 : 0;
        break;
      }
    }
  }
  // Slots that may be left in place with path vertices standing in them: main
  // slots (their candidates are checked one by one) that no later set
  // operation reads and no other slot stands for.
  // leaf_adj: the path vertices that are neighbours of every candidate for
  // vertex n-2, by the operations its slot is made of.
  uint8_t made_of[16] = {1};  // slot 0 is N(v0)
  for (int L = 1; L + 1 < p.nnodes; L++)
    for (int s = p.level_begin[L]; s < (L + 2 < p.nnodes ? p.level_begin[L + 1] : p.nslots); s++) {
      const uint8_t own = d.kind[s] == SLOT_COPY ? 0 : (uint8_t)(1u << L);
      made_of[s] = own | (d.kind[s] == SLOT_FRESH ? 0 : made_of[d.parent[s]]);
      d.hole_ok[s] = !p.labeled && s == p.level_begin[L] && d.alias[s] < 0;
      for (int t = 1; t < p.nslots; t++)
        if ((t != s && d.alias[t] == s) || (d.kind[t] != SLOT_FRESH && d.parent[t] == s)) d.hole_ok[s] = 0;
    }
  if (p.nnodes > 3) d.leaf_adj = made_of[p.level_begin[p.nnodes - 3]];
  // Labeled: the first of the single fresh levels the plan ends in, when there
  // are two of them or more (chain_kernel).
  if (p.labeled && p.nnodes >= 4) {
    int from = p.nnodes - 1;
    for (int L = p.nnodes - 2; L >= 1; L--) {
      const int b = p.level_begin[L], e = L + 2 < p.nnodes ? p.level_begin[L + 1] : p.nslots;
      if (e - b != 1 || d.kind[b] != SLOT_FRESH || __builtin_popcount(p.slot_labels[b]) != 1) break;
      from = L;
    }
    if (from <= p.nnodes - 3) d.chain_from = (int8_t)from;
  }
  // Labeled: levels whose next level only copies (by label) what is there --
  // the search below does not depend on the candidate chosen, so one is
  // searched and counted for all (WarpState::mul).  A six-vertex star on an
  // R-MAT graph of 65,536 vertices and 32 labels, 1.2e10 set operations: 203 ->
  // 0.37 ms (B200).
  if (p.labeled)
    for (int L = 1; L + 2 < p.nnodes; L++) {
      bool copies = true;
      const int e = L + 3 < p.nnodes ? p.level_begin[L + 2] : p.nslots;
      for (int s = p.level_begin[L + 1]; s < e; s++) copies = copies && d.kind[s] == SLOT_COPY;
      if (copies && L + 1 < p.nnodes - 2) d.copy_next |= (uint8_t)(1u << L);
    }
  // The last two levels in one pass (pair_levels): level n-3 is a list of its
  // vertex, or that list met with a slot of the level before, and at most a
  // copy the last slot reads; no bound may involve the last two vertices but
  // the main slot's own.
  const int q2 = p.nnodes - 3;
  if (q2 >= 2) {
    const int b = p.level_begin[q2], k = p.level_begin[q2 + 1] - b, last = d.last_slot;
    const uint32_t early = (1u << q2) - 1u;  // bounds by v_0 .. v_{n-4}
    const bool met = d.kind[b] == SLOT_INTERSECT;
    bool ok = (d.kind[b] == SLOT_FRESH || met) && d.alias[b] < 0;
    if (p.labeled) ok = ok && __builtin_popcount(p.slot_labels[b]) == 1 && __builtin_popcount(p.slot_labels[last]) == 1;
    if (!p.labeled && k == 1 && d.kind[b] == SLOT_COPY && d.alias[b] < 0 && !p.partial[b] && d.kind[last] == SLOT_FRESH &&
        !p.partial[last])
      d.pair = PAIR_SHARED;
    auto within = [&](int small, int large) { return (p.slot_labels[small] & ~p.slot_labels[large]) == 0; };
    if (ok && k == 1) {
      if (d.kind[last] == SLOT_FRESH && !(p.partial[last] & ~early)) d.pair = PAIR_FRESH;
    } else if (ok && k == 2 && d.alias[b + 1] < 0 && d.kind[b + 1] == SLOT_COPY && d.kind[last] != SLOT_FRESH &&
               d.parent[last] == b + 1) {
      const int h = b + 1;
      d.pair_h0 = (int8_t)d.parent[h];
      if (d.kind[last] == SLOT_COPY) {
        if (p.labeled ? within(d.parent[h], h) && within(h, last) : !p.partial[h] && !p.partial[last])
          d.pair = PAIR_COPY;
      } else if (!met && (p.labeled ? within(d.parent[h], h) : !(p.partial[h] & ~early) && !(p.partial[last] & ~early))) {
        d.pair = PAIR_MEET;
      }
    }
  }
  // Cliques (unlabeled, five vertices or more): on every level a main slot
  // that is the prefix of the one helper below the smallest path vertex, both
  // the intersection of the newest vertex's list with the helper before.
  d.clique = !p.labeled && p.nnodes >= 5 && p.partial[0] == 1;
  for (int L = 1; L + 1 < p.nnodes && d.clique; L++) {
    const int b = p.level_begin[L], k = (L + 2 < p.nnodes ? p.level_begin[L + 1] : p.nslots) - b;
    const int up = L == 1 ? 0 : p.level_begin[L - 1] + 1;
    if (k != (L + 2 < p.nnodes ? 2 : 1)) d.clique = 0;
    for (int s = b; s < b + k; s++)
      if (d.kind[s] != SLOT_INTERSECT || d.parent[s] != up || p.partial[s] != (2u << L) - 1u) d.clique = 0;
  }
  // Shape for lane_subtree (unlabeled): level n-3 is one intersection X with
  // a parent at an earlier level, plus at most one alias Y of it; the last
  // slot intersects with X or Y.
  d.l2_x = d.l2_y = -1;
  const int n = p.nnodes;
  if (!p.labeled && n >= 5) {
    const int b = p.level_begin[n - 3], e = p.level_begin[n - 2];
    int x = -1, y = -1, others = 0;
    for (int s = b; s < e; s++) {
      if (d.alias[s] < 0) { if (x < 0) x = s; else others++; }
      else if (y < 0) y = s;
      else others++;
    }
    const int last = d.last_slot;
    if (x >= 0 && !others && (y < 0 || d.alias[y] == x) && d.kind[x] == SLOT_INTERSECT && d.parent[x] < b &&
        d.kind[last] == SLOT_INTERSECT && (d.parent[last] == x || (y >= 0 && d.parent[last] == y))) {
      d.l2_x = (int8_t)x;
      d.l2_y = (int8_t)y;
    }
  }
  return d;
}

RootFilter to_filter(const Plan& p) {
  RootFilter f;
  f.labeled = p.labeled;
  f.need_gt = (!p.labeled && p.partial[0] == 1);
  f.lab0 = p.vertex_label[0];
  f.lab1 = p.vertex_label[1];
  f.d0 = p.degree[0];
  f.d1 = p.degree[1];
  f.d2 = p.degree[2];
  return f;
}

// Parent-set limit of the two-level lane scheme from the run options: 0 =
// default, negative = never, else capped at the shared staging size.  The
// default takes cliques in bit sets first.
constexpr int kLaneSubtreeDefault = 64;
int lane_subtree_limit(const pm_run_opts& o) {
  if (o.lane_subtree_max < 0) return 0;
  return o.lane_subtree_max == 0 ? kLaneSubtreeDefault : std::min(o.lane_subtree_max, PM_SB_MAX);
}

// Whether the tables of a plan's chain (chain_kernel), which are worked out for
// every vertex of a label in each launch, take less time than searching the
// chain below this launch's roots.  How often a root reaches the chain and how
// much is below it grows with the fresh levels of either; measured (B200,
// kernel ms with tables / without, R-MAT, at the start and in the middle of the
// root list), a table costs as much as searching 1 root for every 8 vertices of
// the label where the chain is all and one table deep (4-path: 64M edges on 4M
// vertices, 8 labels, 65,536 roots 1.07 / 0.67 and 1.06 / 0.88, 256 roots 1.03 /
// 0.18 and 1.02 / 0.16; 32 labels, 4,096 roots 0.12 / 0.10); with one such
// level more a single root is worth some 30,000 (4-cycle with a two-vertex
// tail, 8 labels: 1 root 1.57 / 2.64 and 1.05 / 0.33, 16 roots 2.1 / 8.5); with
// two more tables always pay where it matters (5-cycle with the same tail, 1
// root 6.2 / 141 and 1.09 / 0.22).
bool chain_pays(const Plan& p, const DPlan& d, int64_t roots, int64_t label_vertices) {
  if (!d.chain_from) return false;
  int fresh = d.nnodes - 3 - d.chain_from;  // tables but one, then the fresh main slots before the chain
  for (int l = 1; l < d.chain_from; l++) fresh += d.kind[p.level_begin[l]] == SLOT_FRESH;
  return fresh > 1 || roots * (fresh ? 32768 : 8) >= label_vertices;
}

// Worst-case arena words one warp needs for a plan: every materialised slot
// is at most its first operand, itself at most a max-degree list.
int64_t arena_words_for(const Plan& p, int32_t maxdeg, int T) {
  const int64_t per = (T > 0) ? std::min<int64_t>(maxdeg, T) : maxdeg;
  const int materialised = p.nslots - 2;  // minus the root slot and the counted last slot
  return std::max<int64_t>(materialised, 1) * per + 64;
}

}  // namespace

// What a graph keeps per vertex besides its rows, in one allocation (from the
// host: at the end of the rows' own, place_rows -- an allocation and its release
// take longer than the passes that fill it): d_maxnbrdeg, n entries; the two
// 64-bit words in which maxnbrdeg_kernel notes what the lists are like;
// unlabeled in HBM, 33 counts (36 words: of degrees, of rows given out) and
// d_hub_slot.
static size_t maxnbrdeg_bytes(int64_t n) { return sizeof(int32_t) * (size_t)((n + 1) & ~1ll) + 16; }
static bool takes_hub_rows(const pm_graph* g) { return !g->labeled && g->residency == PM_RESIDENT_HBM && g->n > 0; }
static size_t aux_bytes(const pm_graph* g) {
  return maxnbrdeg_bytes(g->n) + (takes_hub_rows(g) ? sizeof(int32_t) * (size_t)(36 + g->n) : 0);
}
static unsigned long long* asym_word(const pm_graph* g) {
  return reinterpret_cast<unsigned long long*>(g->d_maxnbrdeg + ((g->n + 1) & ~1ll));
}

// Bit rows for the vertices with the longest lists: the lowest power of two of a
// degree from 64 on (shorter lists are read as fast as a row) from which all
// rows fit as many bytes as the adjacency array, or 64 MB if that is more, and
// 256 MB at most -- half of them stay in L2.  h[k]: vertices of [2^k, 2^(k+1))
// neighbours.
static void choose_hub_rows(pm_graph* g, const unsigned int* h) {
  const int64_t words = (g->n + 31) / 32;
  const size_t budget = std::min<size_t>(256ull << 20, std::max<size_t>(64ull << 20, 4 * (size_t)g->nadj));
  g->hub_rows = 0;
  g->hub_log = 31;
  for (; g->hub_log > 6 && (g->hub_rows + h[g->hub_log - 1]) * words * 4 <= budget; g->hub_log--)
    g->hub_rows += h[g->hub_log - 1];
}
static size_t hub_bytes(const pm_graph* g) { return g->hub_rows * (size_t)((g->n + 31) / 32) * 4; }

namespace pm {
// Fills g->d_maxnbrdeg from an adjacency array the device can read (HBM or
// mapped host memory).
pm_status compute_maxnbrdeg(pm_graph* g, const int32_t* colidx) {
  if (g->n > 0) {
    PM_CK_PENDING("max neighbour degree");
    CK(cudaMemset(asym_word(g), 0, 16));
    maxnbrdeg_kernel<<<list_blocks(g->n), 512>>>(g->d_rowptr, colidx, g->n, g->d_maxnbrdeg, asym_word(g));
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
  }
  return PM_OK;
}
}  // namespace pm

static pm_status graph_finish(pm_graph* g) {
  // per-vertex max neighbour degree, used by the root filter
  if (!g->d_maxnbrdeg) CK(cudaMalloc(&g->d_maxnbrdeg, aux_bytes(g)));
  g->device_bytes += sizeof(int32_t) * g->n;
  const bool rows_wanted = takes_hub_rows(g) && g->nadj > 0;
  unsigned int* bins = reinterpret_cast<unsigned int*>(asym_word(g) + 2);
  if (g->n > 0 && g->residency == PM_RESIDENT_HBM) {
    PM_CK_PENDING("max neighbour degree");
    CK(cudaMemset(asym_word(g), 0, 16 + (rows_wanted ? 33 * sizeof(unsigned int) : 0)));
    maxnbrdeg_kernel<<<list_blocks(g->n), 512>>>(g->d_rowptr, g->d_colidx, g->n, g->d_maxnbrdeg, asym_word(g));
    CK(cudaGetLastError());
    if (!rows_wanted) CK(cudaDeviceSynchronize());  // (else after the bit rows)
  }
  if (rows_wanted) {
    const int64_t words = (g->n + 31) / 32;
    cudaError_t e = cudaSuccess;
    if (g->hub_log < 0) {  // device arrays: how many rows is not known yet
      unsigned int h[33];
      degree_bins_kernel<<<256, 256>>>(g->d_rowptr, g->n, bins);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpy(h, bins, sizeof(h), cudaMemcpyDeviceToHost);
      if (e == cudaSuccess) choose_hub_rows(g, h);
      if (e == cudaSuccess && g->hub_rows) e = cudaMalloc(&g->d_hub_bits, hub_bytes(g));
      if (e == cudaErrorMemoryAllocation) {  // no room: the graph does without
        (void)cudaGetLastError();
        g->d_hub_bits = nullptr;
        e = cudaSuccess;
      }
    }
    if (e == cudaSuccess && g->d_hub_bits) {
      g->d_hub_slot = reinterpret_cast<int32_t*>(bins + 36);
      e = cudaMemset(g->d_hub_bits, 0, hub_bytes(g));
      if (e == cudaSuccess) {
        hub_rows_kernel<<<list_blocks(g->n), 512>>>(g->d_rowptr, g->d_colidx, g->n, 1 << g->hub_log, words, bins + 32,
                                                    g->d_hub_slot, g->d_hub_bits);
        e = cudaGetLastError();
      }
      g->device_bytes += sizeof(int32_t) * g->n + hub_bytes(g);
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    CK(e);
  }
  if (g->labeled && g->residency == PM_RESIDENT_HBM && g->n > 0) {
    g->nl1 = (g->nlabels > 0 ? g->nlabels : 32) + 1;
    CK(cudaMalloc(&g->d_colidx_lab, sizeof(int32_t) * std::max<int64_t>(g->nadj, 1)));
    CK(cudaMalloc(&g->d_lab_off, sizeof(int32_t) * (size_t)g->n * g->nl1));
    g->device_bytes += sizeof(int32_t) * ((size_t)g->nadj + (size_t)g->n * g->nl1);
    PM_CK_PENDING("label grouping");
    label_group_kernel<<<list_blocks(g->n), 512>>>(g->d_rowptr, g->d_colidx, g->d_labels, 0, g->n, g->nl1, g->d_colidx_lab, 0,
                                      g->d_lab_off);
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
  }
  return PM_OK;
}

// Labeled paged graphs: the label-grouped copy of the adjacency array goes to
// pinned host memory (it is what the frames cache), the group offsets to the
// device.  Grouped on the device from the id-sorted array (h_colidx_dev), a
// vertex range at a time through a bounded device buffer.  With keep_copy
// false only the offsets are kept: the caller's source holds the grouped
// layout already (pm_graph_from_paged_source).
static pm_status paged_group_labels(pm_graph* g, const uint64_t* h_rowptr, bool keep_copy = true) {
  g->nl1 = (g->nlabels > 0 ? g->nlabels : 32) + 1;
  if (keep_copy) {
    CK(cudaHostAlloc((void**)&g->h_colidx_lab, sizeof(int32_t) * std::max<int64_t>(g->nadj, 1),
                     cudaHostAllocMapped | cudaHostAllocPortable));
    CK(cudaHostGetDevicePointer((void**)&g->h_colidx_lab_dev, g->h_colidx_lab, 0));
  }
  CK(cudaMalloc(&g->d_lab_off, sizeof(int32_t) * (size_t)std::max<int64_t>(g->n, 1) * g->nl1));
  g->device_bytes += sizeof(int32_t) * (size_t)g->n * g->nl1;
  const int64_t chunk = std::max<int64_t>(g->maxdeg, std::min<int64_t>(std::max<int64_t>(g->nadj, 1), 64ll << 20));
  int32_t* tmp = nullptr;
  PM_CK_PENDING("label grouping");
  CK(cudaMalloc(&tmp, sizeof(int32_t) * (size_t)std::max<int64_t>(chunk, 1)));
  pm_status st = PM_OK;
  for (int64_t v0 = 0; v0 < g->n && st == PM_OK;) {
    int64_t v1 = v0;
    while (v1 < g->n && (int64_t)(h_rowptr[v1 + 1] - h_rowptr[v0]) <= chunk) v1++;
    const uint64_t b0 = h_rowptr[v0], len = h_rowptr[v1] - b0;
    label_group_kernel<<<list_blocks(v1 - v0), 512>>>(g->d_rowptr, g->h_colidx_dev, g->d_labels, v0, v1, g->nl1, tmp, b0,
                                      g->d_lab_off);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && len && keep_copy)
      e = cudaMemcpy(g->h_colidx_lab + b0, tmp, sizeof(int32_t) * len, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && !keep_copy) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) st = fail(PM_ERR_CUDA, "label grouping: %s", cudaGetErrorString(e));
    v0 = v1;
  }
  cudaFree(tmp);
  if (st != PM_OK) return st;
  if (keep_copy) {
    g->h_paged = g->h_colidx_lab;
    g->h_paged_dev = g->h_colidx_lab_dev;
  }
  return PM_OK;
}

namespace pm {
pm_status paged_place(pm_graph* g, const int32_t* colidx, const pm_graph_opts* o, const int32_t* src_dev);
pm_status paged_maxnbrdeg(pm_graph* g);
void paged_release(pm_graph* g);
pm_status paged_prepare(pm_ctx* ctx, pm_graph* g, bool cold, DPaging* out);
pm_status paged_service_start(pm_ctx* ctx, pm_graph* g);
pm_status paged_service_stop(pm_ctx* ctx, pm_graph* g, pm_stats* st);
int64_t paged_static_frames(const pm_graph* g);
}  // namespace pm

extern "C" void pm_graph_opts_default(pm_graph_opts* o) {
  if (!o) return;
  memset(o, 0, sizeof(*o));
  o->labeled = 0;
  o->device = 0;
  o->residency = PM_RESIDENT_HBM;
  o->page_bytes = 64 * 1024;
  o->frame_pool_bytes = 4ull << 30;
}

// The row offsets and labels of a graph placed from host arrays, on the
// device (every residency).
static pm_status place_rows(pm_graph* g, int64_t n, int64_t nadj, const uint64_t* rowptr, const uint32_t* labels,
                            const pm_graph_opts& o) {
  g->device = o.device;
  g->n = n;
  g->nadj = nadj;
  g->labeled = o.labeled ? 1 : 0;
  g->residency = o.residency;
  int32_t maxd = 0;
  if (takes_hub_rows(g)) {
    unsigned int h[4][32] = {};  // (four of them: neighbours in the array often share a bin)
    for (int64_t v = 0; v < n; v++) {
      const uint32_t d = (uint32_t)(rowptr[v + 1] - rowptr[v]);
      maxd = std::max<int32_t>(maxd, (int32_t)d);
      h[v & 3][31 - __builtin_clz(d | 1u)]++;
    }
    for (int k = 0; k < 32; k++) h[0][k] += h[1][k] + h[2][k] + h[3][k];
    choose_hub_rows(g, h[0]);
  } else {
    for (int64_t v = 0; v < n; v++) maxd = std::max<int32_t>(maxd, (int32_t)(rowptr[v + 1] - rowptr[v]));
  }
  g->maxdeg = maxd;
  CK(cudaMalloc(&g->d_rowptr, sizeof(uint64_t) * (n + 1) + aux_bytes(g)));
  g->d_maxnbrdeg = reinterpret_cast<int32_t*>(g->d_rowptr + n + 1);
  CK(cudaMemcpy(g->d_rowptr, rowptr, sizeof(uint64_t) * (n + 1), cudaMemcpyHostToDevice));
  g->device_bytes += sizeof(uint64_t) * (n + 1);
  if (g->labeled) {
    std::vector<uint8_t> lab((size_t)std::max<int64_t>(n, 1));
    int nl = 0;
    for (int64_t v = 0; v < n; v++) {
      if (labels[v] >= 32) return fail(PM_ERR_FORMAT, "label %u of vertex %lld >= 32", labels[v], (long long)v);
      lab[v] = (uint8_t)labels[v];
      nl = std::max<int>(nl, (int)labels[v] + 1);
    }
    g->nlabels = nl;
    CK(cudaMalloc(&g->d_labels, std::max<int64_t>(n, 1)));
    CK(cudaMemcpy(g->d_labels, lab.data(), n, cudaMemcpyHostToDevice));
    g->device_bytes += n;
  }
  return PM_OK;
}

extern "C" pm_status pm_graph_from_host(int64_t n, int64_t nadj, const uint64_t* rowptr, const int32_t* colidx,
                                        const uint32_t* labels, const pm_graph_opts* opts, pm_graph** out) {
  if (!rowptr || (nadj > 0 && !colidx) || !out || n < 0 || n > INT32_MAX - 1)
    return fail(PM_ERR_INVALID, "pm_graph_from_host: bad arguments");
  pm_graph_opts o;
  pm_graph_opts_default(&o);
  if (opts) o = *opts;
  pm_status st = check_device(o.device);
  if (st != PM_OK) return st;
  if (o.labeled && !labels) return fail(PM_ERR_INVALID, "labeled graph without labels");
  std::unique_ptr<pm_graph> g(new pm_graph);
  st = place_rows(g.get(), n, nadj, rowptr, labels, o);
  if (st != PM_OK) return st;
  if (o.residency == PM_RESIDENT_PAGED) {
    st = paged_place(g.get(), colidx, &o, nullptr);
    if (st != PM_OK) return st;
    g->device_bytes += sizeof(int32_t) * g->n;
    st = paged_maxnbrdeg(g.get());
    if (st != PM_OK) return st;
    if (g->labeled && n > 0) {
      st = paged_group_labels(g.get(), rowptr);
      if (st != PM_OK) return st;
    }
  } else {
    // the adjacency array and, after it, the bit rows (none when memory is short)
    const size_t adj_bytes = (sizeof(int32_t) * (size_t)std::max<int64_t>(nadj, 1) + 255) & ~(size_t)255;
    cudaError_t e = cudaMalloc(&g->d_colidx, adj_bytes + hub_bytes(g.get()));
    if (e == cudaErrorMemoryAllocation && g->hub_rows) {
      (void)cudaGetLastError();
      g->hub_rows = 0;
      e = cudaMalloc(&g->d_colidx, adj_bytes);
    }
    CK(e);
    if (g->hub_rows) g->d_hub_bits = reinterpret_cast<uint32_t*>(g->d_colidx) + adj_bytes / 4;
    if (nadj) CK(cudaMemcpy(g->d_colidx, colidx, sizeof(int32_t) * nadj, cudaMemcpyHostToDevice));
    g->device_bytes += sizeof(int32_t) * nadj;
    st = graph_finish(g.get());
    if (st != PM_OK) return st;
  }
  *out = g.release();
  return PM_OK;
}

extern "C" pm_status pm_graph_from_paged_source(int64_t n, int64_t nadj, const uint64_t* rowptr,
                                                const uint32_t* labels, const int32_t* src, const int32_t* sorted,
                                                const pm_graph_opts* opts, pm_graph** out) {
  if (!rowptr || !out || n < 0 || n > INT32_MAX - 1 || nadj < 0 || (nadj > 0 && !src))
    return fail(PM_ERR_INVALID, "pm_graph_from_paged_source: bad arguments");
  pm_graph_opts o;
  pm_graph_opts_default(&o);
  if (opts) o = *opts;
  o.residency = PM_RESIDENT_PAGED;
  if (o.labeled && (!labels || (nadj > 0 && !sorted)))
    return fail(PM_ERR_INVALID, "a labeled graph needs labels and the id-sorted array");
  if (!o.labeled) sorted = src;
  if (rowptr[n] != (uint64_t)nadj)
    return fail(PM_ERR_INVALID, "rowptr[n] = %llu but n_adj = %lld", (unsigned long long)rowptr[n], (long long)nadj);
  if (((uintptr_t)src & 15) || ((uintptr_t)sorted & 15))
    return fail(PM_ERR_INVALID, "the source arrays must be 16-byte aligned");
  pm_status st = check_device(o.device);
  if (st != PM_OK) return st;
  std::unique_ptr<pm_graph> g(new pm_graph);
  st = place_rows(g.get(), n, nadj, rowptr, labels, o);
  if (st != PM_OK) return st;
  st = paged_place(g.get(), nullptr, &o, src);
  if (st != PM_OK) return st;
  // the id-sorted lists: root filter, features, and a labeled graph's whole
  // lists (read in place)
  g->h_colidx_dev = const_cast<int32_t*>(sorted);
  g->device_bytes += sizeof(int32_t) * g->n;
  st = paged_maxnbrdeg(g.get());
  if (st != PM_OK) return st;
  if (g->labeled && n > 0) {
    st = paged_group_labels(g.get(), rowptr, false);
    if (st != PM_OK) return st;
  }
  *out = g.release();
  return PM_OK;
}

extern "C" pm_status pm_graph_from_device(int64_t n, int64_t nadj, int32_t maxdeg, const uint64_t* d_rowptr,
                                          const int32_t* d_colidx, const uint8_t* d_labels, int device,
                                          pm_graph** out) {
  if (!d_rowptr || (nadj > 0 && !d_colidx) || !out || n < 0 || maxdeg < 0)
    return fail(PM_ERR_INVALID, "pm_graph_from_device: bad arguments");
  pm_status st = check_device(device);
  if (st != PM_OK) return st;
  std::unique_ptr<pm_graph> g(new pm_graph);
  g->device = device;
  g->n = n;
  g->nadj = nadj;
  g->maxdeg = maxdeg;
  g->labeled = d_labels != nullptr;
  g->nlabels = d_labels ? 32 : 0;
  g->owns = false;
  g->d_rowptr = const_cast<uint64_t*>(d_rowptr);
  g->d_colidx = const_cast<int32_t*>(d_colidx);
  g->d_labels = const_cast<uint8_t*>(d_labels);
  st = graph_finish(g.get());
  if (st != PM_OK) return st;
  *out = g.release();
  return PM_OK;
}

extern "C" pm_status pm_graph_open(const char* prefix, const pm_graph_opts* opts, pm_graph** out) {
  pm_graph_opts o;
  pm_graph_opts_default(&o);
  if (opts) o = *opts;
  int64_t n = 0, nadj = 0;
  int32_t maxd = 0;
  uint64_t* rowptr = nullptr;
  int32_t* colidx = nullptr;
  uint32_t* labels = nullptr;
  pm_status st = pm_graph_read(prefix, o.labeled, &n, &nadj, &maxd, &rowptr, &colidx, &labels);
  if (st != PM_OK) return st;
  st = pm_graph_from_host(n, nadj, rowptr, colidx, labels, &o, out);
  free(rowptr);
  free(colidx);
  free(labels);
  return st;
}

extern "C" pm_status pm_graph_get_info(const pm_graph* g, pm_graph_info* info) {
  if (!g || !info) return fail(PM_ERR_INVALID, "pm_graph_get_info: null argument");
  memset(info, 0, sizeof(*info));
  info->n_vertices = g->n;
  info->n_adj = g->nadj;
  info->max_degree = g->maxdeg;
  info->labeled = g->labeled;
  info->n_labels = g->nlabels;
  info->residency = g->residency;
  info->device_bytes = g->device_bytes;
  info->n_pages = (uint64_t)g->n_pages;
  info->n_frames = (uint64_t)g->n_frames;
  info->n_static_frames = (uint64_t)paged_static_frames(g);
  return PM_OK;
}

extern "C" void pm_graph_close(pm_graph* g) {
  if (!g) return;
  cudaSetDevice(g->device);
  if (g->owns) {
    free_dev(g->d_rowptr);
    free_dev(g->d_colidx);
    free_dev(g->d_labels);
  }
  if (!g->owns) {  // else parts of the rows' and the adjacency array's allocations
    free_dev(g->d_maxnbrdeg);
    free_dev(g->d_hub_bits);
  }
  free_dev(g->d_colidx_lab);
  free_dev(g->d_lab_off);
  paged_release(g);
  delete g;
}

extern "C" pm_status pm_ctx_create(int device, pm_ctx** out) {
  if (!out) return fail(PM_ERR_INVALID, "pm_ctx_create: null argument");
  pm_status st = check_device(device);
  if (st != PM_OK) return st;
  std::unique_ptr<pm_ctx> c(new pm_ctx);
  c->device = device;
  CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, device));
  CK(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  CK(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
  for (auto& e : c->ev) CK(cudaEventCreate(&e));
  *out = c.release();
  return PM_OK;
}

extern "C" void* pm_ctx_stream(pm_ctx* c) { return c ? (void*)c->stream : nullptr; }

extern "C" void pm_ctx_destroy(pm_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  cudaStreamSynchronize(c->copy_stream);
  free_dev(c->d_arena);
  free_dev(c->d_ctl);
  if (c->memo) free_dev(c->memo->d);
  delete c->memo;
  free_dev(c->d_feat);
  free_dev(c->d_chain);
  free_dev(c->d_roots);
  free_dev(c->d_tmp);
  free_dev(c->d_vcount);
  free_dev(c->d_voff);
  for (auto& e : c->ev) if (e) cudaEventDestroy(e);
  if (c->stream) cudaStreamDestroy(c->stream);
  if (c->copy_stream) cudaStreamDestroy(c->copy_stream);
  delete c;
}

extern "C" void pm_run_opts_default(pm_run_opts* o) {
  if (!o) return;
  memset(o, 0, sizeof(*o));
  o->root_begin = -1;
  o->root_end = -1;
}

// Builds the root list of plan p into ctx->d_roots + offset; returns count.
static pm_status build_roots(pm_ctx* c, const pm_graph* g, const Plan& p, size_t offset_roots,
                             int64_t* count, bool count_only, int2** roots_buf = nullptr,
                             size_t* roots_bytes = nullptr) {
  if (!roots_buf) { roots_buf = &c->d_roots; roots_bytes = &c->roots_bytes; }
  const int64_t n = g->n;
  if (n == 0) { *count = 0; return PM_OK; }
  if (c->vbuf_n < (size_t)n + 1) {
    free_dev(c->d_vcount);
    free_dev(c->d_voff);
    c->d_vcount = nullptr;
    c->d_voff = nullptr;
    c->vbuf_n = 0;
    CK(cudaMalloc(&c->d_vcount, sizeof(int32_t) * (n + 1)));
    CK(cudaMalloc(&c->d_voff, sizeof(int64_t) * (n + 1)));
    c->vbuf_n = (size_t)n + 1;
  }
  const RootFilter f = to_filter(p);
  const int32_t* colidx = g->residency == PM_RESIDENT_HBM ? g->d_colidx : g->h_colidx_dev;
  PM_CK_PENDING("root filter");
  roots_kernel<false><<<list_blocks(n), 512, 0, c->stream>>>(g->d_rowptr, colidx, g->d_labels, g->d_maxnbrdeg, n, f,
                                                          c->d_vcount, nullptr, nullptr);
  CK(cudaGetLastError());
  CK(cudaMemsetAsync(c->d_vcount + n, 0, sizeof(int32_t), c->stream));
  size_t need = 0;
  CK(cub::DeviceScan::ExclusiveSum(nullptr, need, c->d_vcount, c->d_voff, n + 1, c->stream));
  pm_status st = ensure(&c->d_tmp, &c->tmp_bytes, need);
  if (st != PM_OK) return st;
  CK(cub::DeviceScan::ExclusiveSum(c->d_tmp, need, c->d_vcount, c->d_voff, n + 1, c->stream));
  int64_t total = 0;
  CK(cudaMemcpyAsync(&total, c->d_voff + n, sizeof(int64_t), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  *count = total;
  if (count_only) return PM_OK;
  const size_t want = sizeof(int2) * (offset_roots + (size_t)total) + sizeof(int2);
  if (*roots_bytes < want) {
    // grow, keeping the roots of earlier plans
    int2* nr = nullptr;
    CK(cudaMalloc(&nr, want + want / 4));
    if (*roots_buf && offset_roots)
      CK(cudaMemcpyAsync(nr, *roots_buf, sizeof(int2) * offset_roots, cudaMemcpyDeviceToDevice, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    free_dev(*roots_buf);
    *roots_buf = nr;
    *roots_bytes = want + want / 4;
  }
  PM_CK_PENDING("root filter");
  roots_kernel<true><<<list_blocks(n), 512, 0, c->stream>>>(g->d_rowptr, colidx, g->d_labels, g->d_maxnbrdeg, n, f,
                                                         nullptr, c->d_voff, *roots_buf + offset_roots);
  CK(cudaGetLastError());
  return PM_OK;
}

extern "C" pm_status pm_count_roots(pm_ctx* c, const pm_graph* g, const pm_plan* ph, int64_t* n_roots) {
  if (!c || !g || !ph || !n_roots) return fail(PM_ERR_INVALID, "pm_count_roots: null argument");
  const Plan& p = *plan_of(ph);
  if (p.labeled && !g->labeled) return fail(PM_ERR_INVALID, "labeled plan on an unlabeled graph");
  CK(cudaSetDevice(c->device));
  return build_roots(c, g, p, 0, n_roots, true);
}

namespace pm {
// Root list of one plan in the context's root buffer (valid until the next
// call that builds roots on this context).
pm_status root_list_for(pm_ctx* c, const pm_graph* g, const pm_plan* ph, const int2** roots, int64_t* n) {
  const Plan* p = plan_of(ph);
  if (p->labeled && !g->labeled) return fail(PM_ERR_INVALID, "labeled plan on an unlabeled graph");
  CK(cudaSetDevice(c->device));
  pm_status st = build_roots(c, g, *p, 0, n, false);
  if (st != PM_OK) return st;
  CK(cudaStreamSynchronize(c->stream));
  *roots = c->d_roots;
  return PM_OK;
}

// Exposed for tests through pm_debug_roots: copies the root list of one plan.
pm_status debug_roots(pm_ctx* c, const pm_graph* g, const Plan& p, int32_t* out_pairs, int64_t cap, int64_t* count) {
  pm_status st = build_roots(c, g, p, 0, count, false);
  if (st != PM_OK) return st;
  const int64_t m = std::min<int64_t>(cap, *count);
  if (m > 0) CK(cudaMemcpyAsync(out_pairs, c->d_roots, sizeof(int2) * m, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return PM_OK;
}
}  // namespace pm

extern "C" pm_status pm_debug_roots(pm_ctx* c, const pm_graph* g, const pm_plan* ph, int32_t* out_pairs,
                                    int64_t cap, int64_t* count) {
  if (!c || !g || !ph || !count) return fail(PM_ERR_INVALID, "pm_debug_roots: null argument");
  CK(cudaSetDevice(c->device));
  return debug_roots(c, g, *plan_of(ph), out_pairs, cap, count);
}

// One prepared persistent launch: plans, roots, geometry, kernel arguments.
struct Launch {
  bool labeled = false, paged = false, cold = false, host_copy = false;
  int64_t n_big = 0;          // borrowed arenas
  size_t own_bytes = 0, big_bytes = 0;
  int nplans = 0;
  const Plan* plans[PM_MAX_BATCH];
  DPlan dp[PM_MAX_BATCH];
  MatchArgs a;
  int blocks = 0, threads = 0;
  size_t smem = 0;
  void (*kfn)(const MatchArgs) = nullptr;
  int64_t warps = 0;
  size_t ctl_words = 0;
  int memo_entries = 0;       // per warp (pair_levels)
  std::vector<ChainSteps> chains;  // one per launch of chain_kernel, in order
  std::vector<int> chain_plans;    // steps in each
  const pm_graph* g = nullptr;
};

static constexpr unsigned kDonSlots = 64 * kGroupSlots;  // 64 groups of some 50 warps
// a warp's own arena: at most this many slot words and gather words
static constexpr int64_t kOwnSlotWords = 1 << 16;
static constexpr int64_t kOwnGatherWords = 1 << 15;
static constexpr size_t kBigPoolMaxBytes = 48ull << 30;
static constexpr int kCtlRead = 32 + 32 + kStatWords + 1;  // cursors, counts, stats, status word

// Entries of a warp's value table for a graph of n vertices: one each up to
// 16,384 (a warp's lookups go to the surroundings of a few roots).
static int memo_entries_for(int64_t n) {
  int e = 256;
  while (e < 16384 && e < n) e <<= 1;
  return e;
}

static MemoTables* memo_of(pm_ctx* c) {
  if (!c->memo) c->memo = new MemoTables;
  return c->memo;
}

// Validates the plans and options, builds the root lists into *roots,
// sizes the persistent grid and the arenas, and fills L.  Buffers are grown
// as needed (they belong to the caller: the context for pm_match, the query
// for pm_query_prepare).
static pm_status setup_launch(pm_ctx* c, const pm_graph* g, const pm_plan* const* plans, int nplans,
                              const pm_run_opts& o, int2** roots, size_t* roots_bytes, int32_t** arena,
                              size_t* arena_bytes, unsigned long long** ctl, size_t* ctl_bytes, MemoTables* mt,
                              void** chain, size_t* chain_bytes, Launch* L) {
  if (nplans < 1 || nplans > PM_MAX_BATCH) return fail(PM_ERR_INVALID, "between 1 and %d plans per launch", PM_MAX_BATCH);
  CK(cudaSetDevice(c->device));
  L->labeled = plan_of(plans[0]) && plan_of(plans[0])->labeled != 0;
  for (int i = 0; i < nplans; i++) {
    const Plan* p = plan_of(plans[i]);
    if (!p) return fail(PM_ERR_INVALID, "null plan %d", i);
    if ((p->labeled != 0) != L->labeled) return fail(PM_ERR_INVALID, "plans mix labeled and unlabeled modes");
    if (p->labeled && !g->labeled) return fail(PM_ERR_INVALID, "labeled plan on an unlabeled graph");
    L->plans[i] = p;
  }
  L->nplans = nplans;
  if (o.root_order && nplans != 1) return fail(PM_ERR_INVALID, "root_order needs a single plan");
  const int T = std::max(0, o.truncate);
  const int wpb = o.warps_per_block > 0 ? o.warps_per_block : 8;
  if (wpb > 16 || (wpb & (wpb - 1))) return fail(PM_ERR_INVALID, "warps_per_block must be 1,2,4,8 or 16");
  const int chunk = o.chunk > 0 ? o.chunk : 16;
  const int shard_count = o.shard_count > 1 ? o.shard_count : 1;
  if (o.shard_rank < 0 || o.shard_rank >= shard_count) return fail(PM_ERR_INVALID, "bad shard_rank");
  L->paged = g->residency == PM_RESIDENT_PAGED;
  L->cold = o.cold_cache != 0;
  L->host_copy = o.host_page_copy != 0;

  // root lists, concatenated
  size_t off = 0;
  int64_t arena_words = 64;
  for (int i = 0; i < nplans; i++) {
    const Plan& p = *L->plans[i];
    int64_t cnt = 0;
    pm_status st = build_roots(c, g, p, off, &cnt, false, roots, roots_bytes);
    if (st != PM_OK) return st;
    L->dp[i] = to_dplan(p);
    L->dp[i].nroots = cnt;
    arena_words = std::max(arena_words, arena_words_for(p, g->maxdeg, T));
    off += (size_t)cnt;
  }
  off = 0;
  for (int i = 0; i < nplans; i++) {
    int64_t b = 0, e = L->dp[i].nroots;
    if (o.root_begin >= 0) b = std::min<int64_t>(o.root_begin, e);
    if (o.root_end >= 0) e = std::min<int64_t>(o.root_end, e);
    if (e < b) e = b;
    L->dp[i].roots = *roots + off;
    off += (size_t)L->dp[i].nroots;
    L->dp[i].nroots = e - b;
    L->dp[i].rbase = b;
  }
  // Candidate storage.  worst_* hold every materialised slot at its largest
  // possible size (and, paged, two gathered max-degree lists); each warp's own
  // arena holds that when it is small, else a bounded part of it, and warps
  // that outgrow theirs borrow one of a pool of worst-case arenas.
  const int64_t worst_slots = arena_words;
  const int64_t worst_gather =
      L->paged ? ((std::max<int64_t>(2 * (int64_t)g->maxdeg + 64, 32 * PM_LANE_MAX) + 1) & ~1ll) : 0;
  const int64_t own_slots = std::min<int64_t>(worst_slots, o.own_arena_words > 0 ? o.own_arena_words : kOwnSlotWords);
  const int64_t own_gather =
      L->paged ? ((std::max<int64_t>(std::min<int64_t>(worst_gather, kOwnGatherWords), 32 * PM_LANE_MAX) + 1) & ~1ll)
               : 0;
  const bool borrowing = own_slots < worst_slots || own_gather < worst_gather;
  const int64_t slot_words = own_slots;
  arena_words = own_slots + own_gather;

  // launch geometry: persistent, occupancy-limited
  L->threads = wpb * 32;
  L->smem = sizeof(WarpState) * wpb;
  // kernel variant by register cap: 85 registers (three 256-thread blocks per
  // SM) measures fastest; 16-warp blocks need the uncapped variant
  int variant = o.high_occupancy;
  if (variant == 0) variant = (wpb <= 8) ? 2 : 3;
  if (variant < 0 || variant > 3) return fail(PM_ERR_INVALID, "high_occupancy must be 0..3");
  if ((variant == 1 || variant == 2) && wpb > 8)
    return fail(PM_ERR_INVALID, "warps_per_block 16 needs the uncapped kernel variant (high_occupancy 3)");
  if (variant == 1) {
    L->kfn = L->labeled ? (L->paged ? match_kernel<true, true, 4> : match_kernel<true, false, 4>)
                        : (L->paged ? match_kernel<false, true, 4> : match_kernel<false, false, 4>);
  } else if (variant == 2) {
    L->kfn = L->labeled ? (L->paged ? match_kernel<true, true, 3> : match_kernel<true, false, 3>)
                        : (L->paged ? match_kernel<false, true, 3> : match_kernel<false, false, 3>);
  } else {
    L->kfn = L->labeled ? (L->paged ? match_kernel<true, true, 1> : match_kernel<true, false, 1>)
                        : (L->paged ? match_kernel<false, true, 1> : match_kernel<false, false, 1>);
  }
  int per_sm = 0;
  // per-warp state is ~4 KB: 16-warp blocks need more than the default 48 KB
  CK(cudaFuncSetAttribute(L->kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L->smem));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, L->kfn, L->threads, L->smem));
  if (o.blocks_per_sm > 0) per_sm = std::min(per_sm, o.blocks_per_sm);
  per_sm = std::max(per_sm, 1);
  L->blocks = c->nsm * per_sm;
  L->warps = (int64_t)L->blocks * wpb;
  // keep the arenas within half of the free memory by trimming resident warps
  // (what the buffers of an earlier call hold needs no look at free memory: a
  // query of 50 us spends as much again on asking)
  bool meets = false;
  for (int i = 0; i < nplans; i++)
    meets = meets || (L->dp[i].pair == PAIR_MEET && !L->paged && o.leaf_per_lane == 0 && rows_of_lists(g->maxdeg));
  size_t free_b = 0, total_b = 0;
  const bool fits = !borrowing && (size_t)(L->warps * arena_words * 4) + 256 <= *arena_bytes && *arena &&
                    (!meets || (mt->d && mt->warps == L->warps && mt->entries == memo_entries_for(g->n)));
  if (!fits) {
    CK(cudaMemGetInfo(&free_b, &total_b));
    free_b += *arena_bytes;
  }
  while (!fits && L->blocks > c->nsm && (size_t)(L->warps * arena_words * 4) > free_b / 2) {
    L->blocks -= c->nsm;
    L->warps = (int64_t)L->blocks * wpb;
  }
  // borrowed arenas: as many as a quarter of the free memory holds (capped),
  // at least one, at most one per warp
  const int64_t big_words = borrowing ? worst_slots + worst_gather : 0;
  int64_t n_big = 0;
  if (borrowing) {
    const size_t own_b = (size_t)(L->warps * arena_words * 4);
    const size_t room = free_b / 2 > own_b ? free_b / 2 - own_b : 0;
    const size_t budget = std::min(room / 2, kBigPoolMaxBytes);
    n_big = std::max<int64_t>(1, std::min<int64_t>(L->warps, (int64_t)(budget / ((size_t)big_words * 4))));
    if (o.max_borrowed > 0) n_big = std::min<int64_t>(n_big, o.max_borrowed);
  }
  const size_t own_bytes = (size_t)(L->warps * arena_words * 4);
  const size_t big_bytes = (size_t)n_big * (size_t)big_words * 4;
  pm_status st = ensure((void**)arena, arena_bytes, own_bytes + big_bytes + 4 * (size_t)n_big + 256);
  if (st != PM_OK) return st;
  L->n_big = n_big;
  L->own_bytes = own_bytes;
  L->big_bytes = big_bytes;
  // control block: cursors[32] counts[32] stats[] status sched heartbeat,
  // hand-off ready[] and items[]
  L->ctl_words = 32 + 32 + kStatWords + 24 + (kDonSlots / kGroupSlots) * kSchedStride + kDonSlots + 6 * kDonSlots;
  st = ensure((void**)ctl, ctl_bytes, L->ctl_words * 8);
  if (st != PM_OK) return st;

  // chain tables: one per level of a chain, 32 bytes a vertex, within 1 GiB for
  // the launch (a graph of tens of millions of vertices searches its tails)
  L->g = g;
  if (L->labeled && !L->paged && g->d_lab_off && o.leaf_per_lane == 0 && g->n > 0) {
    const size_t table = sizeof(ulonglong4) * (size_t)g->n;
    size_t need = 0;
    for (int i = 0; i < nplans; i++) {
      if (!chain_pays(*L->plans[i], L->dp[i], L->dp[i].nroots / shard_count, g->n / std::max(1, g->nlabels)))
        L->dp[i].chain_from = 0;
      const size_t levels = L->dp[i].chain_from ? (size_t)(L->dp[i].nnodes - 2 - L->dp[i].chain_from) : 0;
      if (need + levels * table > (1ull << 30)) L->dp[i].chain_from = 0;
      else need += levels * table;
    }
    if (ensure(chain, chain_bytes, need) != PM_OK) {  // no room: the tails are searched
      (void)cudaGetLastError();
      for (int i = 0; i < nplans; i++) L->dp[i].chain_from = 0;
    }
    ulonglong4* at = (ulonglong4*)*chain;
    for (int i = 0; i < nplans; i++) {
      DPlan& d = L->dp[i];
      if (!d.chain_from) continue;
      const Plan& p = *L->plans[i];
      const ulonglong4* next = nullptr;
      size_t step = 0;
      for (int l = d.nnodes - 3; l >= d.chain_from; l--, step++) {
        if (L->chains.size() <= step) {
          L->chains.emplace_back();
          L->chain_plans.push_back(0);
        }
        ChainStep& cs = L->chains[step].s[L->chain_plans[step]++];
        cs.next = next;
        cs.out = at;
        cs.label = p.vertex_label[l];
        cs.part = __builtin_ffs((int)p.slot_labels[p.level_begin[l]]) - 1;
        cs.leaf = __builtin_ffs((int)p.slot_labels[d.last_slot]) - 1;
        next = at;
        at += g->n;
      }
      d.chain = next;
    }
  }

  // value tables for plans that meet lists at the last level: one entry per
  // vertex up to 16,384 (a warp's lookups go to the lists of a few roots'
  // surroundings, not to the whole graph), within an eighth of free memory
  MemoEntry* none = nullptr;
  MemoEntry** memo = &none;
  if (meets) {
    int entries = memo_entries_for(g->n);
    auto need = [&]() { return (size_t)L->warps * (size_t)(entries + 1) * sizeof(MemoEntry); };
    while (!fits && entries > 256 && need() > (free_b + mt->bytes) / 8) entries >>= 1;
    if (fits || need() <= (free_b + mt->bytes) / 8) {
      const bool fresh = mt->bytes < need() || !mt->d;
      if (ensure((void**)&mt->d, &mt->bytes, need()) != PM_OK) {  // no room: lists are walked each time
        (void)cudaGetLastError();
        mt->warps = 0;
      } else {
        if (fresh || mt->warps != L->warps || mt->entries != entries)
          CK(cudaMemsetAsync(mt->d, 0, need(), c->stream));
        mt->warps = L->warps;
        mt->entries = entries;
        L->memo_entries = entries;
        memo = &mt->d;
      }
    }
  }

  MatchArgs& a = L->a;
  memset(&a, 0, sizeof(a));
  a.rowptr = g->d_rowptr;
  a.colidx = g->d_colidx;
  a.labels = g->d_labels;
  a.colidx_lab = g->d_colidx_lab;
  a.lab_off = g->d_lab_off;
  // plans whose last two levels this launch does not take in one pass
  // (truncated: an unlabeled list's first T elements less the path vertices
  // among them is not its length less them)
  for (int i = 0; i < nplans; i++) {
    uint8_t& pair = L->dp[i].pair;
    if (o.leaf_per_lane != 0 || (L->labeled ? !g->d_lab_off : L->paged) ||
        (!L->labeled && T && (pair == PAIR_FRESH || pair == PAIR_SHARED)) || (pair == PAIR_MEET && (L->paged || !*memo)))
      pair = PAIR_NONE;
  }
  a.asym = g->n > 0 ? asym_word(g) : nullptr;
  a.memo = *memo;
  a.memo_entries = L->memo_entries;
  a.hub_slot = g->d_hub_slot;
  a.hub_bits = g->d_hub_bits;
  a.hub_words = (int32_t)((g->n + 31) / 32);
  a.host_sorted = (g->residency == PM_RESIDENT_PAGED && g->d_lab_off) ? g->h_colidx_dev : nullptr;
  a.leaf_flat = o.leaf_per_lane == 1 || !rows_of_lists(g->maxdeg) ? 0 : (o.leaf_per_lane == 2 ? 2 : 1);
  a.lane_subtree_max = lane_subtree_limit(o);
  a.clique_bits = a.lane_subtree_max == kLaneSubtreeDefault;
  a.nl1 = g->nl1;
  a.n = (int32_t)g->n;
  a.nplans = nplans;
  a.T = T;
  a.chunk = chunk;
  // Unless the caller sets the pop size, a pop is as many roots as leave every
  // warp eight pops (one at least, the shard unit at most): sixteen roots per
  // pop left a query of 2,000 roots to 120 of 3,552 warps (the 4-clique on 400
  // vertices: 225 us of kernel).
  int64_t total_roots = 0;
  for (int i = 0; i < nplans; i++) total_roots += L->dp[i].nroots / shard_count;
  a.pop = o.chunk > 0 ? chunk : (int32_t)std::max<int64_t>(1, std::min<int64_t>(chunk, total_roots / (8 * L->warps)));
  a.shard_rank = o.shard_rank;
  a.shard_count = shard_count;
  a.split_min = o.split_level1 == 0 ? 64 : (o.split_level1 < 0 ? 0 : o.split_level1);
  a.maxdeg = g->maxdeg;
  unsigned long long* w = *ctl;
  a.cursors = w; w += 32;
  a.counts = w; w += 32;
  a.stats = w; w += kStatWords;
  a.status = (unsigned int*)w; w += 1;
  a.all_sched = w; w += 1;
  a.started = (unsigned int*)w; w += 1;
  a.heartbeat = w; w += 21;
  a.don_groups = kDonSlots / kGroupSlots;
  a.sched = w; w += a.don_groups * kSchedStride;
  a.don_ready = w; w += kDonSlots;
  a.don_items = (int4*)w; w += 6 * kDonSlots;
  a.total_warps = (unsigned int)L->warps;
  a.arena = *arena;
  a.arena_words = arena_words;
  a.slot_words = slot_words;
  a.gather_words = arena_words - slot_words;
  a.n_big = (int32_t)n_big;
  a.big_arena = n_big ? (int32_t*)((char*)*arena + own_bytes) : nullptr;
  a.big_slot_words = worst_slots;
  a.big_gather_words = worst_gather;
  a.big_owner = n_big ? (unsigned int*)((char*)*arena + own_bytes + big_bytes) : nullptr;
  a.root_counts = (unsigned long long*)o.root_counts;
  a.root_cost = o.root_cost;
  a.root_reads = o.root_reads;
  a.root_order = o.root_order;
  if (o.root_split && nplans != 1) return fail(PM_ERR_INVALID, "root_split needs a single plan");
  a.root_split = o.root_split;
  a.timeout_ns = (unsigned long long)(o.timeout_ms > 0 ? o.timeout_ms : 600000) * 1000000ull;
  if (o.prefetch_off || o.prefetch_pages || o.prefetch_chunks) {
    if (!L->paged) return fail(PM_ERR_INVALID, "prefetch lists need a paged graph");
    if (nplans != 1 || !o.prefetch_off || !o.prefetch_pages || o.prefetch_chunks < 0)
      return fail(PM_ERR_INVALID, "prefetch lists need one plan, both arrays and a chunk count");
    a.pf_off = o.prefetch_off;
    a.pf_pages = o.prefetch_pages;
    a.pf_chunks = o.prefetch_chunks;
    a.pf_ahead = o.prefetch_ahead > 0 ? o.prefetch_ahead : 2;
  }
  for (int i = 0; i < nplans; i++) a.plans[i] = L->dp[i];
  if (L->paged) {
    st = paged_prepare(c, const_cast<pm_graph*>(g), L->cold, &a.pg);
    if (st != PM_OK) return st;
    a.pg.dev_copy = L->host_copy ? 0 : 1;
  }
  return PM_OK;
}

// Enqueues one launch on the context stream: control reset, the persistent
// kernel (its plans travel in its parameter block) between events eb/ee, and
// the read-back of counts, stats and status into host_ctl.  Capturable into a
// CUDA graph (host_ctl must then be pinned).
static pm_status enqueue_launch(pm_ctx* c, Launch& L, unsigned long long* host_ctl, cudaEvent_t eb, cudaEvent_t ee) {
  // everything up to the hand-off items, which are written before they are read
  CK(cudaMemsetAsync(L.a.cursors, 0, (size_t)((char*)L.a.don_items - (char*)L.a.cursors), c->stream));
  if (L.n_big) CK(cudaMemsetAsync(L.a.big_owner, 0, 4 * (size_t)L.n_big, c->stream));
  if (eb) CK(cudaEventRecord(eb, c->stream));
  PM_CK_PENDING("pm_match");
  for (size_t k = 0; k < L.chains.size(); k++) {
    const pm_graph* g = L.g;
    const dim3 grid((unsigned)std::min<int64_t>((g->n + 255) / 256, 1024), (unsigned)L.chain_plans[k]);
    chain_kernel<<<grid, 256, 0, c->stream>>>(L.chains[k], g->d_rowptr, g->d_colidx_lab, g->d_lab_off, g->nl1,
                                              g->d_labels, g->n, L.a.T);
  }
  L.kfn<<<L.blocks, L.threads, L.smem, c->stream>>>(L.a);
  CK(cudaGetLastError());
  if (ee) CK(cudaEventRecord(ee, c->stream));
  CK(cudaMemcpyAsync(host_ctl, L.a.cursors, sizeof(unsigned long long) * kCtlRead, cudaMemcpyDeviceToHost,
                     c->stream));
  return PM_OK;
}

// Turns the read-back control words into counts, stats and a status.
static pm_status finish_launch(const Launch& L, const unsigned long long* host_ctl, float kernel_ms, float roots_ms,
                               const pm_stats& pst, uint64_t* counts_out, pm_stats* stats_out) {
  const unsigned int status = (unsigned int)(host_ctl[64 + kStatWords] & 0xffffffffu);
  for (int i = 0; i < L.nplans; i++) {
    const Plan& p = *L.plans[i];
    counts_out[i] = host_ctl[32 + i] * (p.labeled ? 1ull : (uint64_t)p.multiplicity);
  }
  if (stats_out) {
    pm_stats& so = *stats_out;
    so = pst;
    const unsigned long long* stt = host_ctl + 64;
    so.set_ops = stt[ST_SETOPS];
    so.alg_bytes = stt[ST_BYTES];
    so.n_roots = stt[ST_ROOTS];
    so.splits = stt[ST_SPLITS];
    so.page_hits = stt[ST_HITS];
    so.page_misses = stt[ST_MISSES];
    so.zero_copy_bytes = stt[ST_ZC_BYTES];
    so.evictions = stt[ST_EVICTIONS];
    so.warp_ns = stt[ST_WARP_NS];
    so.idle_ns = stt[ST_IDLE_NS];
    so.kernel_ms = kernel_ms;
    so.roots_ms = roots_ms;
    so.grid_blocks = L.blocks;
    so.block_threads = L.threads;
    so.arena_bytes = (uint64_t)(L.own_bytes + L.big_bytes);
    so.borrowed_arenas = stt[ST_BORROWS];
    so.leaf_cycles = stt[ST_LEAF_CYC];
    so.level_cycles = stt[ST_LEVEL_CYC];
    so.prefix_cycles = stt[ST_PREFIX_CYC];
    so.prefetch_requests = stt[ST_PREFETCH];
    so.page_requests = stt[ST_REQUESTS];
    so.page_dropped = stt[ST_DROPPED];
    so.device_page_loads = stt[ST_DEV_LOADS];
    so.pages_loaded += stt[ST_DEV_LOADS];  // the service thread's count plus the warps'
    so.h2d_page_bytes += stt[ST_DEV_BYTES];
    so.arena_pool = (uint64_t)L.n_big;
    so.device_status = status;
  }
  if (status & DEV_ARENA_OVERFLOW) return fail(PM_ERR_INTERNAL, "device: candidate set exceeded the warp arena");
  if (status & DEV_TIMEOUT) return fail(PM_ERR_TIMEOUT, "device: the launch hit its time limit or a bounded wait gave up");
  if (status) return fail(PM_ERR_INTERNAL, "device status 0x%x", status);
  return PM_OK;
}

// Runs an enqueued launch to completion, with the page service around it.
template <class Enqueue>
static pm_status run_launch(pm_ctx* c, const pm_graph* g, Launch& L, Enqueue enqueue, pm_stats* pst) {
  memset(pst, 0, sizeof(*pst));
  if (L.paged) {
    pm_status st = paged_service_start(c, const_cast<pm_graph*>(g));
    if (st != PM_OK) return st;
  }
  pm_status est = enqueue();
  cudaError_t sync_err = cudaStreamSynchronize(c->stream);
  if (L.paged) {
    pm_status sst = paged_service_stop(c, const_cast<pm_graph*>(g), pst);
    if (sst != PM_OK && est == PM_OK && sync_err == cudaSuccess) return sst;
  }
  if (est != PM_OK) return est;
  CK(sync_err);
  return PM_OK;
}

extern "C" pm_status pm_match(pm_ctx* c, const pm_graph* g, const pm_plan* const* plans, int nplans,
                              const pm_run_opts* opts, uint64_t* counts_out, pm_stats* stats_out) {
  if (!c || !g || !plans || nplans < 1 || !counts_out) return fail(PM_ERR_INVALID, "pm_match: bad arguments");
  pm_run_opts o;
  pm_run_opts_default(&o);
  if (opts) o = *opts;
  CK(cudaSetDevice(c->device));
  cudaEvent_t e0 = c->ev[0], e1 = c->ev[1], e2 = c->ev[2];
  CK(cudaEventRecord(e0, c->stream));
  std::unique_ptr<Launch> L(new Launch);
  pm_status st = setup_launch(c, g, plans, nplans, o, &c->d_roots, &c->roots_bytes, &c->d_arena, &c->arena_bytes,
                              &c->d_ctl, &c->ctl_bytes, memo_of(c), &c->d_chain, &c->chain_bytes, L.get());
  if (st != PM_OK) return st;
  unsigned long long host_ctl[kCtlRead];
  pm_stats pst;
  st = run_launch(c, g, *L, [&]() { return enqueue_launch(c, *L, host_ctl, e1, e2); }, &pst);
  if (st != PM_OK) return st;
  float kms = 0, rms = 0;
  CK(cudaEventElapsedTime(&kms, e1, e2));
  CK(cudaEventElapsedTime(&rms, e0, e1));
  return finish_launch(*L, host_ctl, kms, rms, pst, counts_out, stats_out);
}

// ---------------------------------------------------------------------
// Prepared queries: the root lists, arenas and launch sequence are built
// once; each run replays the launch captured in a CUDA graph.
// ---------------------------------------------------------------------
struct pm_query {
  pm_ctx* c = nullptr;
  const pm_graph* g = nullptr;
  Launch L;
  int2* d_roots = nullptr;
  size_t roots_bytes = 0;
  int32_t* d_arena = nullptr;
  size_t arena_bytes = 0;
  unsigned long long* d_ctl = nullptr;
  size_t ctl_bytes = 0;
  MemoTables memo;
  void* d_chain = nullptr;
  size_t chain_bytes = 0;
  unsigned long long* h_ctl = nullptr;  // pinned
  cudaEvent_t eb = nullptr, ee = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  float roots_ms = 0;
};

extern "C" void pm_query_free(pm_query* q) {
  if (!q) return;
  cudaSetDevice(q->c->device);
  if (q->exec) cudaGraphExecDestroy(q->exec);
  if (q->graph) cudaGraphDestroy(q->graph);
  if (q->eb) cudaEventDestroy(q->eb);
  if (q->ee) cudaEventDestroy(q->ee);
  free_dev(q->d_roots);
  free_dev(q->d_arena);
  free_dev(q->d_ctl);
  free_dev(q->memo.d);
  free_dev(q->d_chain);
  if (q->h_ctl) cudaFreeHost(q->h_ctl);
  delete q;
}

extern "C" pm_status pm_query_prepare(pm_ctx* c, const pm_graph* g, const pm_plan* const* plans, int nplans,
                                      const pm_run_opts* opts, pm_query** out) {
  if (!c || !g || !plans || !out) return fail(PM_ERR_INVALID, "pm_query_prepare: bad arguments");
  pm_run_opts o;
  pm_run_opts_default(&o);
  if (opts) o = *opts;
  CK(cudaSetDevice(c->device));
  std::unique_ptr<pm_query, void (*)(pm_query*)> q(new pm_query, pm_query_free);
  q->c = c;
  q->g = g;
  CK(cudaEventRecord(c->ev[0], c->stream));
  pm_status st = setup_launch(c, g, plans, nplans, o, &q->d_roots, &q->roots_bytes, &q->d_arena, &q->arena_bytes,
                              &q->d_ctl, &q->ctl_bytes, &q->memo, &q->d_chain, &q->chain_bytes, &q->L);
  if (st != PM_OK) return st;
  CK(cudaEventRecord(c->ev[1], c->stream));
  CK(cudaEventSynchronize(c->ev[1]));
  CK(cudaEventElapsedTime(&q->roots_ms, c->ev[0], c->ev[1]));
  CK(cudaMallocHost(&q->h_ctl, sizeof(unsigned long long) * kCtlRead));
  CK(cudaEventCreate(&q->eb));
  CK(cudaEventCreate(&q->ee));
  CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  // timing events stay outside the graph (recorded around each replay)
  pm_status est = enqueue_launch(c, q->L, q->h_ctl, nullptr, nullptr);
  cudaError_t cerr = cudaStreamEndCapture(c->stream, &q->graph);
  if (est != PM_OK) return est;
  CK(cerr);
  CK(cudaGraphInstantiate(&q->exec, q->graph, 0));
  *out = q.release();
  return PM_OK;
}

extern "C" pm_status pm_query_run(pm_query* q, uint64_t* counts_out, pm_stats* stats_out) {
  if (!q || !counts_out) return fail(PM_ERR_INVALID, "pm_query_run: bad arguments");
  pm_ctx* c = q->c;
  CK(cudaSetDevice(c->device));
  if (q->L.paged) {
    DPaging pg;
    pm_status st = paged_prepare(c, const_cast<pm_graph*>(q->g), q->L.cold, &pg);  // reset the page table
    if (st != PM_OK) return st;
  }
  pm_stats pst;
  pm_status st = run_launch(c, q->g, q->L, [&]() -> pm_status {
    CK(cudaEventRecord(q->eb, c->stream));
    CK(cudaGraphLaunch(q->exec, c->stream));
    CK(cudaEventRecord(q->ee, c->stream));
    return PM_OK;
  }, &pst);
  if (st != PM_OK) return st;
  float kms = 0;
  CK(cudaEventElapsedTime(&kms, q->eb, q->ee));
  return finish_launch(q->L, q->h_ctl, kms, q->roots_ms, pst, counts_out, stats_out);
}

// ---------------------------------------------------------------------
// Allocation-free entry point: pm_match_static.
//
// For callers that must not allocate device memory -- code running while
// another library holds the device allocator lock, in a process whose
// allocator is owned by a framework with a fixed pool, or in a service that
// has budgeted every byte up front.  The caller provides the graph arrays
// and receives the count; everything the launch needs besides them (control
// block, donation ring, root list, per-warp arenas) lives in one file-scope
// device array of PM_STATIC_SCRATCH_BYTES that each GPU keeps from module
// load until the process exits.  The plan travels in the kernel's parameter
// block like every launch's, so the scratch is the only state it shares.
// ---------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_scratch[PM_STATIC_SCRATCH_BYTES];

namespace {
// Donation slots inside the static scratch (with the groups' words no more
// than 4,096 slots and one set of words took before).
constexpr unsigned kStaticRing = 8 * kGroupSlots;
constexpr size_t kStaticCtlWords =
    32 + 32 + kStatWords + 24 + (kStaticRing / kGroupSlots) * kSchedStride + kStaticRing + 6 * kStaticRing;

struct StaticScratch {
  bool ready = false;
  unsigned char* base = nullptr;  // device address of g_static_scratch on this device
};
StaticScratch g_static[64];
std::mutex g_static_mu;

// Root filter with unordered, bounded compaction (no scan, no temporary
// buffer): each warp reserves slots with one atomic per 32 edges; writes past
// `cap` are skipped and the host sees the true total afterwards.  The 2-hop
// test scans the neighbour's list for a vertex of sufficient degree.
__global__ void roots_static_kernel(const uint64_t* rowptr, const int32_t* colidx, const uint8_t* labels, int64_t n,
                                    RootFilter f, int2* out, unsigned long long cap, unsigned long long* counter) {
  const int lane = lane_id();
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
    const uint64_t b = rowptr[r], e = rowptr[r + 1];
    if ((long long)(e - b) < f.d0 || (f.labeled && labels[r] != f.lab0)) continue;
    for (uint64_t i0 = b; i0 < e; i0 += 32) {
      const uint64_t i = i0 + lane;
      bool keep = false;
      int c = 0;
      if (i < e) {
        c = colidx[i];
        keep = (!f.need_gt || r > c) && (!f.labeled || labels[c] == f.lab1) &&
               (int)(rowptr[c + 1] - rowptr[c]) >= f.d1;
        if (keep) {
          bool two_hop = false;
          for (uint64_t d = rowptr[c]; d < rowptr[c + 1] && !two_hop; d++) {
            const int u = colidx[d];
            two_hop = (int)(rowptr[u + 1] - rowptr[u]) >= f.d2;
          }
          keep = two_hop;
        }
      }
      const unsigned bal = __ballot_sync(FULL, keep);
      unsigned long long base = 0;
      if (lane == 0 && bal) base = atomicAdd(counter, (unsigned long long)__popc(bal));
      base = __shfl_sync(FULL, base, 0);
      if (keep) {
        const unsigned long long pos = base + __popc(bal & lanemask_lt());
        if (pos < cap) out[pos] = make_int2((int)r, c);
      }
    }
  }
}
}  // namespace

extern "C" pm_status pm_match_static(const uint64_t* d_rowptr, const int32_t* d_colidx, const uint8_t* d_labels,
                                     int64_t n, int64_t nadj, int32_t max_degree, const pm_plan* plan,
                                     const pm_run_opts* opts, void* stream, uint64_t* count_out,
                                     pm_stats* stats_out) {
  if (!d_rowptr || (nadj > 0 && !d_colidx) || !plan || !count_out || n < 0 || max_degree < 0)
    return fail(PM_ERR_INVALID, "pm_match_static: bad arguments");
  if (n > INT32_MAX - 1) return fail(PM_ERR_INVALID, "pm_match_static: %lld vertices exceed int32 ids", (long long)n);
  const Plan& p = *plan_of(plan);
  if (p.labeled && !d_labels) return fail(PM_ERR_INVALID, "pm_match_static: labeled plan without labels");
  pm_run_opts o;
  pm_run_opts_default(&o);
  if (opts) o = *opts;
  if (o.root_counts || o.root_cost || o.root_reads || o.root_order || o.root_split || o.shard_count > 1 ||
      o.root_begin >= 0 || o.root_end >= 0 || o.prefetch_off || o.prefetch_pages || o.prefetch_chunks)
    return fail(PM_ERR_INVALID,
                "pm_match_static: per-root inputs and outputs, root orders, ranges, shards and prefetch lists are not "
                "supported");
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(PM_ERR_INVALID, "pm_match_static: device %d out of range", dev);
  cudaStream_t st = (cudaStream_t)stream;
  // set-up, once per device, with that device current
  unsigned char* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static[dev].ready) {
      unsigned char* ptr = nullptr;
      cudaError_t e = cudaGetSymbolAddress((void**)&ptr, g_static_scratch);
      if (e != cudaSuccess)
        return fail(PM_ERR_CUDA, "pm_match_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      g_static[dev].base = ptr;
      g_static[dev].ready = true;
    }
    base = g_static[dev].base;
  }
  int nsm = 0;
  CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int T = std::max(0, o.truncate);
  const int wpb = o.warps_per_block > 0 ? o.warps_per_block : 8;
  if (wpb > 16 || (wpb & (wpb - 1)))
    return fail(PM_ERR_INVALID, "pm_match_static: warps_per_block must be 1,2,4,8 or 16");
  const int64_t slot_words = arena_words_for(p, max_degree, T);
  const size_t warp_bytes = (size_t)slot_words * 4;
  const size_t ctl_bytes = kStaticCtlWords * 8;
  const size_t min_arena = (size_t)wpb * warp_bytes;  // one block
  if (ctl_bytes + 64 + min_arena + 256 > PM_STATIC_SCRATCH_BYTES)
    return fail(PM_ERR_INVALID,
                "pm_match_static: one block of warp arenas needs %zu bytes, beyond the %llu-byte static scratch "
                "(max degree %d is too large for this entry point)",
                min_arena, (unsigned long long)PM_STATIC_SCRATCH_BYTES, max_degree);
  // layout: control block | root counter | roots | arenas
  unsigned long long* ctl = (unsigned long long*)base;
  unsigned long long* rcount = (unsigned long long*)(base + ctl_bytes);
  int2* roots = (int2*)(base + ctl_bytes + 64);
  const size_t after_ctl = PM_STATIC_SCRATCH_BYTES - ctl_bytes - 64;
  const unsigned long long root_cap = (after_ctl - min_arena - 256) / sizeof(int2);

  CK(cudaMemsetAsync(base, 0, ctl_bytes + 64, st));  // previous calls leave their contents behind
  const RootFilter f = to_filter(p);
  PM_CK_PENDING("pm_match_static");
  roots_static_kernel<<<4 * nsm, 256, 0, st>>>(d_rowptr, d_colidx, d_labels, n, f, roots, root_cap, rcount);
  CK(cudaGetLastError());
  unsigned long long nroots = 0;
  CK(cudaMemcpyAsync(&nroots, rcount, sizeof(nroots), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (nroots > root_cap)
    return fail(PM_ERR_INVALID, "pm_match_static: %llu root edges exceed the %llu the static scratch holds",
                nroots, root_cap);
  const size_t roots_bytes = ((size_t)nroots * sizeof(int2) + 255) & ~(size_t)255;
  int32_t* arena = (int32_t*)((unsigned char*)roots + roots_bytes);
  // 256 bytes of slack after the last arena: bulk copies of a slot round its
  // end up to 16 bytes
  const size_t arena_bytes = after_ctl - roots_bytes - 256;
  // kernel variant by register cap, as pm_match chooses it
  int variant = o.high_occupancy;
  if (variant == 0) variant = (wpb <= 8) ? 2 : 3;
  if (variant < 0 || variant > 3) return fail(PM_ERR_INVALID, "pm_match_static: high_occupancy must be 0..3");
  if ((variant == 1 || variant == 2) && wpb > 8)
    return fail(PM_ERR_INVALID, "pm_match_static: warps_per_block 16 needs the uncapped kernel variant");
  void (*kfn)(const MatchArgs) =
      variant == 1 ? (p.labeled ? match_kernel<true, false, 4> : match_kernel<false, false, 4>)
      : variant == 2 ? (p.labeled ? match_kernel<true, false, 3> : match_kernel<false, false, 3>)
                     : (p.labeled ? match_kernel<true, false, 1> : match_kernel<false, false, 1>);
  int per_sm = 0;
  CK(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(WarpState) * wpb)));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, wpb * 32, sizeof(WarpState) * wpb));
  if (o.blocks_per_sm > 0) per_sm = std::min(per_sm, o.blocks_per_sm);
  int64_t blocks = std::max(1, per_sm) * (int64_t)nsm;
  blocks = std::min<int64_t>(blocks, (int64_t)(arena_bytes / ((size_t)wpb * warp_bytes)));
  if (blocks < 1) return fail(PM_ERR_INTERNAL, "pm_match_static: no room for a block of arenas");

  DPlan dp = to_dplan(p);
  dp.pair = PAIR_NONE;  // (no symmetry words, label groups or value tables here)
  dp.roots = roots;
  dp.nroots = (int64_t)nroots;
  MatchArgs a;
  memset(&a, 0, sizeof(a));
  a.plans[0] = dp;
  a.rowptr = d_rowptr;
  a.colidx = d_colidx;
  a.labels = d_labels;
  a.leaf_flat = o.leaf_per_lane == 1 || !rows_of_lists(max_degree) ? 0 : (o.leaf_per_lane == 2 ? 2 : 1);
  a.lane_subtree_max = lane_subtree_limit(o);
  a.clique_bits = a.lane_subtree_max == kLaneSubtreeDefault;
  a.n = (int32_t)n;
  a.nplans = 1;
  a.T = T;
  a.chunk = o.chunk > 0 ? o.chunk : 16;
  a.pop = o.chunk > 0 ? o.chunk
                      : (int32_t)std::max<int64_t>(1, std::min<int64_t>(16, (int64_t)nroots / (8 * blocks * wpb)));
  a.shard_rank = 0;
  a.shard_count = 1;
  a.split_min = o.split_level1 == 0 ? 64 : (o.split_level1 < 0 ? 0 : o.split_level1);
  a.maxdeg = max_degree;
  unsigned long long* w = ctl;
  a.cursors = w; w += 32;
  a.counts = w; w += 32;
  a.stats = w; w += kStatWords;
  a.status = (unsigned int*)w; w += 1;
  a.all_sched = w; w += 1;
  a.started = (unsigned int*)w; w += 1;
  a.heartbeat = w; w += 21;
  a.don_groups = kStaticRing / kGroupSlots;
  a.sched = w; w += a.don_groups * kSchedStride;
  a.don_ready = w; w += kStaticRing;
  a.don_items = (int4*)w; w += 6 * kStaticRing;
  const int64_t warps = blocks * wpb;
  a.total_warps = (unsigned int)warps;
  a.arena = arena;
  a.arena_words = slot_words;
  a.slot_words = slot_words;
  a.gather_words = 0;
  a.n_big = 0;
  a.timeout_ns = (unsigned long long)(o.timeout_ms > 0 ? o.timeout_ms : 600000) * 1000000ull;
  PM_CK_PENDING("pm_match_static");
  kfn<<<(int)blocks, wpb * 32, sizeof(WarpState) * wpb, st>>>(a);
  CK(cudaGetLastError());
  unsigned long long host_ctl[kCtlRead];
  CK(cudaMemcpyAsync(host_ctl, ctl, sizeof(host_ctl), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  Launch L;
  L.nplans = 1;
  L.plans[0] = &p;
  L.own_bytes = (size_t)warps * (size_t)slot_words * 4;
  L.blocks = (int)blocks;
  L.threads = wpb * 32;
  L.warps = warps;
  L.a = a;
  pm_stats pst;
  memset(&pst, 0, sizeof(pst));
  return finish_launch(L, host_ctl, 0.f, 0.f, pst, count_out, stats_out);
}
