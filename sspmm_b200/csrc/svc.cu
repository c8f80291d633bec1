// Sparse vector compression kernels.
//
// Reference behaviour (RowMerge/sparse_matrix_format.py:100-123): for vector row i,
//     cols = []
//     for j in 0..V-1 (rows below M only):  cols = list(set(cols + row[V*i+j]))
// and the vector row pointer is the running sum of len(cols).  The order of `cols`
// is CPython's set order, which for small non-negative ints is decided by an
// open-addressing table: hash(x) = x; start slot x & mask; probe the nine following
// slots when that window fits inside the table, else jump to (5*i + 1 + perturb) & mask
// with perturb >>= 5; after an insertion with 5*fill >= 3*mask the table is rebuilt
// with the power-of-two length above 4*used (2*used beyond 50 000), re-inserting
// the old entries in slot order; iteration is in slot order.
//
// A "team" (one warp, or one CTA) works on one vector row; the V rows of a group
// are one contiguous CSR range.
//   svc_count_kernel   marks the group's columns in a shared-memory bitmap with
//                      atomicOr, counts first-time bits by popc of the returned
//                      words, and decides per group whether ascending order is
//                      already the exact answer: it is when the largest column id
//                      is below the final table length (every key then sits in its
//                      home slot).
//   svc_scan_*         exclusive scans (vector row pointers, scratch offsets) and a
//                      histogram of replay classes.
//   svc_emit_sorted    bitmap -> ascending column list by a popc prefix scan; value
//                      vectors placed with prefix[word] + popc(lower bits).
//   svc_emit_replay    exact replay of the V set rebuilds.  Insertion into a table of
//                      fixed length is "first come, first served" along each key's
//                      probe path, which has a unique fixed point: slot = the first
//                      one on my path not held by an earlier element.  The team finds
//                      it in parallel with atomic minima on words that hold the element's
//                      sequence number and its column; table growth steps are replayed
//                      level by level (8, 32, 128, ...).  Small tables are filled in batches
//                      of the sequence whose losers go on in rounds (BitTable,
//                      insert_batches); the tables of large sets are kept from one rebuild
//                      to the next, which starts from them (relevel).
//                      Stack of 16 power-law matrices (n 4096 to 65536, V = 8), whole
//                      call: 877 us; 1033 with every small table filled by all elements at
//                      once, 3080 to 3450 also with free tables at every rebuild.  Per launch,
//                      classes L, M2, M1, S, XS 613, 454, 276, 189, 199 us one after another
//                      (600, 503, 436, 228, 286 before batches).
// The replay kernels take their groups from per-class lists (written by the scan kernel)
// through a work counter, so a CTA never walks over groups of other classes and the
// groups of a class, whose cost differs by an order of magnitude, balance themselves.
#include "svc.cuh"

#include <mutex>
#include <type_traits>

#include "launch.h"
#include "ptx.cuh"

namespace sspmm_b200 {

__device__ int g_svc_bad_column = 0;

namespace {

constexpr int kMinTable = 8;
constexpr int kLinearProbes = 9;
constexpr int kPerturbShift = 5;

// Replay classes by number of distinct columns u (and final table length):
constexpr int kClassSorted = 0;   // no replay
constexpr int kClassS = 1;        // u <= 306   (table <= 512):   warp team, everything in shared memory
constexpr int kClassM1 = 2;       // u <= 1228  (table <= 2048):  CTA team, everything in shared memory
constexpr int kClassM2 = 3;       // u <= 4914  (table <= 8192):  CTA team, everything in shared memory
constexpr int kClassL = 4;        // table <= 32768:              CTA team, table in shared memory, lists in global
constexpr int kClassXL = 5;       // larger:                      CTA team, table and lists in global
constexpr int kClassXS = 6;       // u <= 76    (table <= 128):   warp team, small enough for 48 resident teams per SM
constexpr int kNumClasses = kSvcClasses;
static_assert(kNumClasses == 7, "class numbering");

constexpr int kXSCapU = 76, kXSCapT = 128;
constexpr int kSCapU = 306, kSCapT = 512;
constexpr int kM1CapU = 1228, kM1CapT = 2048;
constexpr int kM2CapU = 4914, kM2CapT = 8192;
constexpr int kLCapT = 32768;
constexpr int kLCapU = 19660;   // most keys a table of kLCapT slots holds

__host__ __device__ inline void next_level(int size, long long& trig, int& next_size) {
    const long long mask = size - 1;
    trig = (3 * mask + 4) / 5;                         // smallest fill with 5*fill >= 3*mask
    const long long minused = trig > 50000 ? trig * 2 : trig * 4;
    long long ns = kMinTable;
    while (ns <= minused) ns <<= 1;
    next_size = (int)(ns > (1ll << 30) ? (1ll << 30) : ns);
}

// Table length after `distinct` different keys were added to an empty set.
__host__ __device__ inline int final_table_len(int distinct) {
    int size = kMinTable;
    for (;;) {
        long long trig;
        int ns;
        next_level(size, trig, ns);
        if (distinct < trig || size >= (1 << 30)) return size;
        size = ns;
    }
}

__host__ __device__ inline int replay_class(int u, int tbl_len) {
    if (tbl_len <= 0) return kClassSorted;
    if (u <= kXSCapU) return kClassXS;
    if (u <= kSCapU) return kClassS;
    if (u <= kM1CapU) return kClassM1;
    if (u <= kM2CapU) return kClassM2;
    if (tbl_len <= kLCapT) return kClassL;
    return kClassXL;
}

// The list of replayed groups is written segment by segment.  A segment is a class, or a part of one: the groups
// of a class differ in cost by the ratio of their sizes (up to four), and with only a few groups per team the order
// in which the work counter hands them out decides how long the last team runs.  So the classes with few, long
// groups are cut into four size ranges (two for S) that are listed largest first.
constexpr int kNumSegs = kSvcSegs;
constexpr int kSegS = 1, kSegM1 = 3, kSegM2 = 7, kSegL = 11, kSegXL = 15, kSegXS = 16, kSegSortedBig = 17;
static_assert(kNumSegs == 18, "segment numbering");
// Groups in ascending order with more than kBigGroup entries get a CTA each; the counting pass marks them
// (table length -1) and the last segment lists them.
__host__ __device__ inline int size_quarter(int u, int cap) {       // 0 = the largest sizes of a class whose largest is cap
    if (u > (int)((long long)cap * 181 / 256)) return 0;            // cap / sqrt(2)
    if (u > cap / 2) return 1;
    if (u > (int)((long long)cap * 91 / 256)) return 2;             // cap / (2 sqrt(2))
    return 3;
}
__host__ __device__ inline int list_segment(int u, int tbl_len) {
    switch (replay_class(u, tbl_len)) {
        case kClassS: return kSegS + (u > kSCapU / 2 ? 0 : 1);
        case kClassM1: return kSegM1 + size_quarter(u, kM1CapU);
        case kClassM2: return kSegM2 + size_quarter(u, kM2CapU);
        case kClassL: return kSegL + size_quarter(u, kLCapU);
        case kClassXL: return kSegXL;
        case kClassXS: return kSegXS;
        default: return tbl_len < 0 ? kSegSortedBig : 0;
    }
}
// first segment of a class and one past its last
__host__ inline void class_segments(int c, int& s0, int& s1) {
    switch (c) {
        case kClassS: s0 = kSegS; s1 = kSegM1; break;
        case kClassM1: s0 = kSegM1; s1 = kSegM2; break;
        case kClassM2: s0 = kSegM2; s1 = kSegL; break;
        case kClassL: s0 = kSegL; s1 = kSegXL; break;
        case kClassXL: s0 = kSegXL; s1 = kSegXS; break;
        case kClassXS: s0 = kSegXS; s1 = kSegSortedBig; break;
        default: s0 = 0; s1 = 1; break;
    }
}

// Global scratch ints of one replayed group: a list of class L, class XL's table and two lists.
__host__ __device__ inline long long group_scratch_ints(int u, int tbl_len) {
    const int c = replay_class(u, tbl_len);
    if (c == kClassL) return ((long long)u + 3) & ~3ll;
    if (c == kClassXL) return ((2ll * u + 3) & ~3ll) + tbl_len;
    return 0;
}

__device__ __forceinline__ int warp_sum(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// ---- teams -------------------------------------------------------------------
struct WarpTeam {
    static constexpr int kSize = 32;
    static constexpr int kPerBlock = 8;
    __device__ static int tid() { return threadIdx.x & 31; }
    __device__ static int index_in_block() { return threadIdx.x >> 5; }
    __device__ static void sync() { __syncwarp(); }
    __device__ static int sum(int v, int*) { return warp_sum(v); }
    __device__ static int max_of(int v, int*) { return warp_max(v); }
    __device__ static int broadcast(int v, int*) { return __shfl_sync(0xffffffffu, v, 0); }   // value of thread 0
};

template <int THREADS>
struct BlockTeam {
    static constexpr int kSize = THREADS;
    [[maybe_unused]] static constexpr int kPerBlock = 1;
    __device__ static int tid() { return threadIdx.x; }
    __device__ static int index_in_block() { return 0; }
    __device__ static void sync() { __syncthreads(); }
    __device__ static bool any(bool p, int*) { return __syncthreads_or(p ? 1 : 0) != 0; }
    __device__ static int sum(int v, int* scratch) {            // scratch: 33 ints of shared memory
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
        __syncthreads();
        int t = 0;
        for (int w = 0; w < THREADS / 32; ++w) t += scratch[w];
        __syncthreads();
        return t;
    }
    __device__ static int max_of(int v, int* scratch) {
        v = warp_max(v);
        if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
        __syncthreads();
        int t = scratch[0];
        for (int w = 1; w < THREADS / 32; ++w) t = max(t, scratch[w]);
        __syncthreads();
        return t;
    }
    __device__ static int broadcast(int v, int* scratch) {     // value of thread 0
        if (threadIdx.x == 0) scratch[32] = v;
        __syncthreads();
        const int r = scratch[32];
        __syncthreads();
        return r;
    }
    // sum of the warps' numbers (the same in every lane) before this warp, and of all; scratch: 32 ints, free until the next barrier
    __device__ static int before(int count, int& total, int* scratch) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane == 0) scratch[warp] = count;
        __syncthreads();
        const int v = lane < THREADS / 32 ? scratch[lane] : 0;
        const int incl = warp_incl_scan(v, lane);
        total = __shfl_sync(0xffffffffu, incl, 31);
        return __shfl_sync(0xffffffffu, incl - v, warp);
    }
};

// Groups with many entries get a whole CTA, the others a warp: two launches of the same kernel,
// each taking the groups that pass its filter (0 = all, 1 = at most kBigGroup entries, 2 = more).
constexpr int kBigGroup = 1024;
constexpr int kBigTeam = 1024;             // threads of such a CTA
// Where every group gets a CTA it has 1024 threads as long as all are resident at once, else 256: with 2250 groups of 256 to 8000 entries
// the larger ones took 116 to 131 us a call, 60 to 72 now (59 to 75 before groups got 1024 threads), with 256 groups of 37 k entries
// (V = 16) 108 against 125.  Those of 256 have to fill an SM's threads, with at most 32 registers (1000 groups of 18 k entries: 271 us
// with 40, 241 with 32); those of 1024 are faster with what they take (the large groups of a stack of 16: 60 us, 62.5 with 32).
constexpr int kTeam = 256;
__device__ __forceinline__ bool group_passes(int filter, int entries) {
    return filter == 0 || (filter == 1) == (entries <= kBigGroup);
}

// ---------------------------------------------------------------- pass 1: count
constexpr int kLookAt = 64;
template <class Team>
__global__ void __launch_bounds__(Team::kSize * Team::kPerBlock, 2048 / (Team::kSize * Team::kPerBlock))
svc_count_kernel(SvcProblem p, int words, int filter, int* __restrict__ counts, int* __restrict__ mode,
                 int* __restrict__ tbl_len) {
    extern __shared__ unsigned int sm_words[];
    __shared__ int red[33], found[kLookAt], n_found;
    unsigned int* bm = sm_words + (size_t)Team::index_in_block() * words;
    const int tid = Team::tid();
    auto count_group = [&](int i) {
        const int r0 = min(i * p.V, p.M), r1 = min(i * p.V + p.V, p.M);
        const int e0 = p.row_ptr[r0], e1 = p.row_ptr[r1];
        if (!group_passes(filter, e1 - e0)) return;
        const int* const cols = p.col_idx + e0;
        const unsigned n_entries = (unsigned)max(0, e1 - e0);             // (an entry's number may come within a step of 2^31)
        if (e1 - e0 < words) {
            for (unsigned e = tid; e < n_entries; e += Team::kSize) {
                const unsigned c = (unsigned)cols[e];
                if (c < (unsigned)p.K) bm[c >> 5] = 0u;
            }
        } else {
            for (int w = tid; w < words; w += Team::kSize) bm[w] = 0u;
        }
        Team::sync();
        int cnt = 0, mx = -1, bad = 0;
        for (unsigned e = tid; e < n_entries; e += 4 * Team::kSize) {      // four loads in flight
            int c4[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) c4[b] = e + b * Team::kSize < n_entries ? cols[e + b * Team::kSize] : -1;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int c = c4[b];
                if ((unsigned)c < (unsigned)p.K) {
                    const unsigned bit = 1u << (c & 31);
                    const unsigned old = atomicOr(&bm[c >> 5], bit);
                    cnt += (old & bit) ? 0 : 1;
                    mx = max(mx, c);
                } else if (e + b * Team::kSize < n_entries) {
                    bad = 1;
                }
            }
        }
        cnt = Team::sum(cnt, red);
        mx = Team::max_of(mx, red);
        bad = Team::max_of(bad, red);
        if (tid == 0) {
            counts[i] = cnt;
            const int len = final_table_len(cnt);
            const int replay = (mx >= len) ? 1 : 0;
            mode[i] = replay;
            tbl_len[i] = replay ? len : ((e1 - e0) > kBigGroup ? -1 : 0);     // -1: ascending order, and large enough for a CTA
            if (bad) g_svc_bad_column = 1;
        }
        Team::sync();
    };
    if (Team::kPerBlock == 1 && filter == 2) {
        // the large groups are few: a CTA looks at kLookAt groups at a time, a thread each (one after another, the look-ups of a stack
        // of 45 k groups took 296 CTAs 90 us)
        for (int first = blockIdx.x * kLookAt; first < p.m_vec; first += gridDim.x * kLookAt) {
            if (tid == 0) n_found = 0;
            __syncthreads();
            const int i = first + tid;
            if (tid < kLookAt && i < p.m_vec &&
                group_passes(2, p.row_ptr[min(i * p.V + p.V, p.M)] - p.row_ptr[min(i * p.V, p.M)])) found[atomicAdd(&n_found, 1)] = i;
            __syncthreads();
            const int n = n_found;
            for (int x = 0; x < n; ++x) count_group(found[x]);
            __syncthreads();
        }
        return;
    }
    for (int i = blockIdx.x * Team::kPerBlock + Team::index_in_block(); i < p.m_vec; i += gridDim.x * Team::kPerBlock) count_group(i);
}

// ---------------------------------------------------------------- scans
// Exclusive scans over the groups (vector row pointers from the counts, scratch offsets) and the lists of replayed
// groups per class, in three small launches: per-block sums, a scan of the block sums by one CTA, and the final
// positions; matrices of one block (4096 groups) do it all in the last one.  A block covers kScanBlock groups; a block
// sum is kScanFields numbers: vectors, scratch ints, and the groups of each list segment.
// What bounds these kernels is their barriers: the segments are counted with shared-memory atomics and only the two sums
// are reduced across the block.  (Reducing all twenty fields block-wide took 19 + 24 + 33 us whatever the size.)  Inside a
// segment the groups are listed in no particular order; the lists only say who works on what.
// totals: [0] nvec, [1] scratch ints, [2..2+kNumSegs) groups per list segment, then the bad-column flag
constexpr int kScanThreads = 1024;
constexpr int kScanPerThread = 4;
constexpr int kScanBlock = kScanThreads * kScanPerThread;
constexpr int kScanFields = 2 + kNumSegs;
static_assert(kScanFields == kSvcScanFields, "scan fields");

// Exclusive prefixes of a and b over the threads of the block, in thread order, and their totals.  sh: 2 x 32 long longs.
__device__ __forceinline__ void block_prefix_pair(long long& a, long long& b, long long& total_a, long long& total_b, long long (*sh)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long ta = __shfl_up_sync(0xffffffffu, ia, o), tb = __shfl_up_sync(0xffffffffu, ib, o);
        if (lane >= o) { ia += ta; ib += tb; }
    }
    if (lane == 31) { sh[0][warp] = ia; sh[1][warp] = ib; }
    __syncthreads();
    // every warp scans the warp totals for itself
    long long wa = sh[0][lane], wb = sh[1][lane];
    const long long own_a = wa, own_b = wb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long ta = __shfl_up_sync(0xffffffffu, wa, o), tb = __shfl_up_sync(0xffffffffu, wb, o);
        if (lane >= o) { wa += ta; wb += tb; }
    }
    total_a = __shfl_sync(0xffffffffu, wa, 31);
    total_b = __shfl_sync(0xffffffffu, wb, 31);
    a = ia - a + __shfl_sync(0xffffffffu, wa - own_a, warp);
    b = ib - b + __shfl_sync(0xffffffffu, wb - own_b, warp);
}

// A thread's groups: counts, scratch and segments (-1 past the end).  Segments with list entries are counted into `seg`.
struct ScanItems {
    int u[kScanPerThread], cls[kScanPerThread], rank[kScanPerThread];
    long long scr[kScanPerThread], vectors = 0, scratch = 0;
    __device__ __forceinline__ void load(int m_vec, const int* counts, const int* tbl_len, int* seg) {
        const int first = blockIdx.x * kScanBlock + threadIdx.x * kScanPerThread;
        int len[kScanPerThread];
#pragma unroll
        for (int j = 0; j < kScanPerThread; ++j) {
            u[j] = first + j < m_vec ? counts[first + j] : 0;
            len[j] = first + j < m_vec ? tbl_len[first + j] : 0;
        }
#pragma unroll
        for (int j = 0; j < kScanPerThread; ++j) {
            cls[j] = -1; scr[j] = 0; rank[j] = 0;
            if (first + j >= m_vec) continue;
            scr[j] = group_scratch_ints(u[j], len[j]);
            cls[j] = list_segment(u[j], len[j]);
            vectors += u[j];
            scratch += scr[j];
        }
        // one atomic per segment and warp: most groups of a matrix are in one or two segments
#pragma unroll
        for (int j = 0; j < kScanPerThread; ++j) {
            const unsigned peers = __match_any_sync(0xffffffffu, cls[j]);
            const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
            int base = 0;
            if (lane == leader && cls[j] >= 0) base = atomicAdd(&seg[cls[j]], __popc(peers));
            rank[j] = __shfl_sync(0xffffffffu, base, leader) + __popc(peers & ((1u << lane) - 1u));
        }
    }
};

__global__ void __launch_bounds__(kScanThreads)
svc_scan_sums_kernel(int m_vec, const int* __restrict__ counts, const int* __restrict__ tbl_len,
                     long long* __restrict__ block_sums) {
    __shared__ long long sh[2][32];
    __shared__ int seg[kNumSegs];
    if (threadIdx.x < kNumSegs) seg[threadIdx.x] = 0;
    __syncthreads();
    ScanItems it;
    it.load(m_vec, counts, tbl_len, seg);
    long long a = it.vectors, b = it.scratch, total_a, total_b;
    block_prefix_pair(a, b, total_a, total_b, sh);          // its barrier also completes the segment counts
    long long* mine = block_sums + (size_t)blockIdx.x * kScanFields;
    if (threadIdx.x == 0) { mine[0] = total_a; mine[1] = total_b; }
    if (threadIdx.x < kNumSegs) mine[2 + threadIdx.x] = seg[threadIdx.x];
}

// One CTA: block_sums -> exclusive prefixes in place, and the totals; a warp per field.
__global__ void __launch_bounds__(32 * kScanFields)
svc_scan_blocks_kernel(int n_blocks, long long* __restrict__ block_sums, long long* __restrict__ totals, long long* __restrict__ host_totals) {
    const int field = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long carry = 0;
    for (int b0 = 0; b0 < n_blocks; b0 += 32) {
        const int b = b0 + lane;
        const long long v = b < n_blocks ? block_sums[(size_t)b * kScanFields + field] : 0;
        long long inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (b < n_blocks) block_sums[(size_t)b * kScanFields + field] = carry + inc - v;
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) {
        totals[field] = carry;
        if (host_totals) host_totals[field] = carry;
    }
    if (threadIdx.x == 0) {
        totals[kScanFields] = g_svc_bad_column;          // reported with the totals, then cleared
        if (host_totals) host_totals[kScanFields] = g_svc_bad_column;
        g_svc_bad_column = 0;
    }
}

// vec_ptr: counts in, exclusive scan out (and the total at [m_vec]); tbl_off: scratch offsets; class_list: the
// replayed groups segment by segment (see list_segment).  ALONE: the only block, which also writes the totals.
template <bool ALONE>
__global__ void __launch_bounds__(kScanThreads)
svc_scan_place_kernel(int m_vec, int* __restrict__ vec_ptr, const int* __restrict__ tbl_len,
                      long long* __restrict__ tbl_off, const long long* __restrict__ block_sums,
                      long long* __restrict__ totals, long long* __restrict__ host_totals, int* __restrict__ class_list) {
    __shared__ long long sh[2][32];
    __shared__ int seg[kNumSegs], seg_at[kNumSegs];
    if (threadIdx.x < kNumSegs) seg[threadIdx.x] = 0;
    __syncthreads();
    ScanItems it;
    it.load(m_vec, vec_ptr, tbl_len, seg);
    long long a = it.vectors, b = it.scratch, total_a, total_b;
    block_prefix_pair(a, b, total_a, total_b, sh);          // its barrier also completes the segment counts
    // where segment k starts in the list: after all groups of the segments before it (segment 0 is not replayed)
    if (threadIdx.x < 32) {
        const int k = threadIdx.x;
        const int groups = k >= 1 && k < kNumSegs ? (ALONE ? seg[k] : (int)totals[2 + k]) : 0;
        const int start = warp_incl_scan(groups, k) - groups;
        if (k < kNumSegs) seg_at[k] = start + (ALONE ? 0 : (int)block_sums[(size_t)blockIdx.x * kScanFields + 2 + k]);
    }
    __syncthreads();
    if (!ALONE) {
        a += block_sums[(size_t)blockIdx.x * kScanFields];
        b += block_sums[(size_t)blockIdx.x * kScanFields + 1];
    }
    const int first = blockIdx.x * kScanBlock + threadIdx.x * kScanPerThread;
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
        const int i = first + j;
        if (i >= m_vec) break;
        vec_ptr[i] = (int)a;
        tbl_off[i] = b;
        a += it.u[j];
        b += it.scr[j];
        if (it.cls[j] > 0) class_list[seg_at[it.cls[j]] + it.rank[j]] = i;
    }
    if (ALONE) {
        auto report = [&](int field, long long v) {
            totals[field] = v;
            if (host_totals) host_totals[field] = v;
        };
        if (threadIdx.x < kNumSegs) report(2 + threadIdx.x, seg[threadIdx.x]);
        if (threadIdx.x == 0) {
            report(0, total_a);
            report(1, total_b);
            vec_ptr[m_vec] = (int)total_a;
            tbl_off[m_vec] = total_b;
            report(kScanFields, g_svc_bad_column);           // reported with the totals, then cleared
            g_svc_bad_column = 0;
        }
    } else if (blockIdx.x == 0 && threadIdx.x == 0) {
        vec_ptr[m_vec] = (int)totals[0];
        tbl_off[m_vec] = totals[1];
    }
}

// ---------------------------------------------------------------- pass 2a: ascending order
// Zeroes the value vectors of a group; the team's barrier before the values are put in.
template <class Team>
__device__ __forceinline__ void zero_values(__half* out_vals, int64_t base, int n, int V) {
    uint4* dst = reinterpret_cast<uint4*>(out_vals + base * V);
    for (int x = Team::tid(); x < n * (V / 8); x += Team::kSize) dst[x] = make_uint4(0, 0, 0, 0);
}
// Row ends of a group in shared memory: rows[0 .. n_rows].
constexpr int kRowInts = 20;
// The matrix row (inside the group) of entry e.
__device__ __forceinline__ int row_of_entry(const int* rows, int n_rows, int e) {
    int r = 0;
#pragma unroll
    for (int step = 8; step > 0; step >>= 1)
        if (r + step < n_rows && e >= rows[r + step]) r += step;
    return r;
}
// Calls f(row, column, value) for the group's entries, four in flight per thread.
template <class Team, class F>
__device__ __forceinline__ void for_each_value(const SvcProblem& p, const int* rows, int n_rows, F&& f) {
    const int e0 = rows[0];
    const int* const cols = p.col_idx + e0;
    const __half* const vals = p.vals + e0;
    const unsigned n_entries = (unsigned)max(0, rows[n_rows] - e0);
    for (unsigned e = Team::tid(); e < n_entries; e += 4 * Team::kSize) {
        int c[4];
        __half v[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const unsigned x = e + b * Team::kSize;
            c[b] = x < n_entries ? cols[x] : -1;
            v[b] = x < n_entries ? vals[x] : __half(0);
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if ((unsigned)c[b] < (unsigned)p.K) f(row_of_entry(rows, n_rows, (int)(e0 + e + b * Team::kSize)), c[b], v[b]);
    }
}

// Bound by the latency of its look-ups, so the large groups get 1024 threads and every thread four entries at a time (conv weight of
// 512 x 4608, 64 groups: 14.7 us with 256 threads and an entry each, 10.6 now, zeroing included).
template <class Team>
__global__ void __launch_bounds__(Team::kSize * Team::kPerBlock, Team::kSize == kTeam ? 2048 / kTeam : 1)
svc_emit_sorted_kernel(SvcProblem p, int words, int filter, const int* __restrict__ vec_ptr,
                       const int* __restrict__ mode, int* __restrict__ out_ptr, int* __restrict__ out_col, __half* __restrict__ out_vals,
                       const int* __restrict__ list, int n_list) {
    extern __shared__ unsigned int sm_words[];
    __shared__ int red[33], all_rows[Team::kPerBlock * kRowInts];
    unsigned int* bm = sm_words + (size_t)Team::index_in_block() * words * 2;
    unsigned int* pre = bm + words;
    int* const rows = all_rows + Team::index_in_block() * kRowInts;
    const int tid = Team::tid(), lane = tid & 31;
    // with a list: only the groups it names; else every group
    const int n_loop = list ? n_list : p.m_vec;
    for (int k = blockIdx.x * Team::kPerBlock + Team::index_in_block(); k < n_loop; k += gridDim.x * Team::kPerBlock) {
        const int i = list ? list[k] : k;
        if (out_ptr && tid == 0) {
            out_ptr[i] = vec_ptr[i];
            if (i == p.m_vec - 1) out_ptr[p.m_vec] = vec_ptr[p.m_vec];
        }
        if (mode[i] != 0) continue;
        const int r0 = min(i * p.V, p.M), n_rows = min(i * p.V + p.V, p.M) - r0;
        const int e0 = p.row_ptr[r0], e1 = p.row_ptr[r0 + n_rows];
        const int base = vec_ptr[i];
        if (e1 == e0 || !group_passes(filter, e1 - e0)) continue;
        if (tid <= n_rows) rows[tid] = p.row_ptr[r0 + tid];
        for (int w = tid; w < words; w += Team::kSize) bm[w] = 0u;
        if (out_vals && p.zero_values) zero_values<Team>(out_vals, base, vec_ptr[i + 1] - base, p.V);
        Team::sync();
        const int* const cols = p.col_idx + e0;
        const unsigned n_entries = (unsigned)max(0, e1 - e0);
        for (unsigned e = tid; e < n_entries; e += 4 * Team::kSize) {
            int c[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) c[b] = e + b * Team::kSize < n_entries ? cols[e + b * Team::kSize] : -1;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if ((unsigned)c[b] < (unsigned)p.K) atomicOr(&bm[c[b] >> 5], 1u << (c[b] & 31));
        }
        Team::sync();
        // columns by a lane per bit when the words are well filled (a thread per word would write up to 32 of them in turn)
        const bool by_bit = Team::kSize >= 256 && (e1 - e0) >= 8 * words;
        int running = 0;
        for (int w0 = 0; w0 < words; w0 += Team::kSize) {
            const int w = w0 + tid;
            unsigned word = (w < words) ? bm[w] : 0u;
            const int pc = __popc(word);
            // exclusive prefix of pc over the team, in thread order
            int incl = warp_incl_scan(pc, lane);
            int chunk_total;
            if constexpr (Team::kSize == 32) {
                chunk_total = __shfl_sync(0xffffffffu, incl, 31);
            } else {
                incl += Team::before(__shfl_sync(0xffffffffu, incl, 31), chunk_total, red);
                Team::sync();
            }
            int o = running + incl - pc;
            if (w < words) pre[w] = (unsigned)o;
            o += base;
            while (word && !by_bit) {
                const int b = __ffs(word) - 1;
                out_col[o++] = w * 32 + b;
                word &= word - 1;
            }
            running += chunk_total;
        }
        Team::sync();
        if (by_bit) {
#pragma unroll 4
            for (int w = tid >> 5; w < words; w += Team::kSize / 32) {
                const unsigned word = bm[w];
                if ((word >> lane) & 1u) out_col[base + (int)pre[w] + __popc(word & ((1u << lane) - 1u))] = w * 32 + lane;
            }
        }
        if (out_vals)
            for_each_value<Team>(p, rows, n_rows, [&](int r, int c, __half v) {
                const int pos = (int)pre[c >> 5] + __popc(bm[c >> 5] & ((1u << (c & 31)) - 1u));
                out_vals[((int64_t)base + pos) * p.V + r] = v;
            });
        Team::sync();
    }
}

// ---------------------------------------------------------------- pass 2b: hash-table replay
struct Probe {            // position on a key's probe path
    unsigned i;           // start of the current window
    unsigned w;           // offset inside the window
    unsigned perturb;
};
__device__ __forceinline__ Probe probe_begin(unsigned key, unsigned mask) {
    Probe p;
    p.i = key & mask; p.w = 0; p.perturb = key;
    return p;
}
__device__ __forceinline__ void probe_advance(Probe& p, unsigned mask) {
    const unsigned window = (p.i + kLinearProbes <= mask) ? kLinearProbes : 0;
    if (p.w < window) {
        ++p.w;
        return;
    }
    p.perturb >>= kPerturbShift;
    p.i = (p.i * 5u + 1u + p.perturb) & mask;
    p.w = 0;
}
// Growth of a set's table (next_level in closed form for the lengths that occur, at most 2^19).
__device__ __forceinline__ int level_trigger(int size) { return (3 * (size - 1) + 4) / 5; }       // the fill that makes it grow
__device__ __forceinline__ int level_next(int size) { return size > 65536 ? size * 2 : size * 4; }

// Position of a slot on a key's probe path.
__device__ __forceinline__ Probe probe_at(unsigned key, unsigned mask, unsigned slot) {
    Probe p = probe_begin(key, mask);
    const unsigned ahead = slot - p.i;
    if (ahead <= kLinearProbes && (ahead == 0 || p.i + kLinearProbes <= mask)) {       // in the window of its home slot, as nearly all are
        p.w = ahead;
        return p;
    }
    for (unsigned n = 0; p.i + p.w != slot && n <= 8u * mask + 64u; ++n) probe_advance(p, mask);
    return p;
}

constexpr unsigned kFree = 0xffffffffu;          // word of a free slot

struct SharedWords {
    uint32_t at;
    __device__ __forceinline__ SharedWords part(unsigned i) const { return SharedWords{at + 4u * i}; }
    __device__ __forceinline__ unsigned ld(unsigned i) const {
        unsigned v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at + 4u * i) : "memory");
        return v;
    }
    __device__ __forceinline__ void st(unsigned i, unsigned v) const { asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + 4u * i), "r"(v) : "memory"); }
    __device__ __forceinline__ void free4(unsigned i) const {
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at + 4u * i), "r"(kFree) : "memory");
    }
    __device__ __forceinline__ unsigned take(unsigned i, unsigned v) const {       // atomic minimum, the word before
        unsigned old;
        asm volatile("atom.shared.min.u32 %0, [%1], %2;" : "=r"(old) : "r"(at + 4u * i), "r"(v) : "memory");
        return old;
    }
    __device__ __forceinline__ void claim(unsigned i, unsigned v) const { asm volatile("red.shared.min.u32 [%0], %1;" ::"r"(at + 4u * i), "r"(v) : "memory"); }
    __device__ __forceinline__ void set(unsigned i, unsigned v) const { asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(at + 4u * i), "r"(v) : "memory"); }
    __device__ __forceinline__ bool give_up(unsigned i, unsigned v) const {        // frees the slot if it still holds v
        unsigned old;
        asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;" : "=r"(old) : "r"(at + 4u * i), "r"(v), "r"(kFree) : "memory");
        return old == v;
    }
};
struct GlobalWords {
    unsigned* at;
    __device__ __forceinline__ GlobalWords part(unsigned i) const { return GlobalWords{at + i}; }
    __device__ __forceinline__ unsigned ld(unsigned i) const { return __ldcg(at + i); }
    __device__ __forceinline__ void st(unsigned i, unsigned v) const { __stcg(at + i, v); }
    __device__ __forceinline__ void free4(unsigned i) const { __stcg(reinterpret_cast<uint4*>(at + i), make_uint4(kFree, kFree, kFree, kFree)); }
    __device__ __forceinline__ unsigned take(unsigned i, unsigned v) const { return atomicMin(at + i, v); }
    __device__ __forceinline__ void claim(unsigned i, unsigned v) const { atomicMin(at + i, v); }
    __device__ __forceinline__ bool give_up(unsigned i, unsigned v) const { return atomicCAS(at + i, v, kFree) == v; }
};

// A list that only the CTA that owns it touches: its reads may come from L1.
struct GlobalList {
    unsigned* at;
    __device__ __forceinline__ unsigned ld(unsigned i) const {
        unsigned v;
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(at + i) : "memory");
        return v;
    }
    __device__ __forceinline__ void st(unsigned i, unsigned v) const { asm volatile("st.global.u32 [%0], %1;" ::"l"(at + i), "r"(v) : "memory"); }
};

// A bit per slot that is taken; a word more than the table needs, since windows are read as two words.
// to_free: to the first free slot on the path from position p on (a table is never more than 60 % full, and the jumps reach every slot).
__device__ __forceinline__ void to_free(const SharedWords& bits, Probe& p, unsigned mask) {
    for (;;) {
        const unsigned at = p.i >> 5;
        const unsigned window = __funnelshift_r(bits.ld(at), bits.ld(at + 1), p.i & 31u);
        const unsigned open = ~window & (p.i + kLinearProbes <= mask ? (2u << kLinearProbes) - 1u : 1u) & (~0u << p.w);
        if (open) {
            p.w = __ffs(open) - 1;
            return;
        }
        p.perturb >>= kPerturbShift;
        p.i = (p.i * 5u + 1u + p.perturb) & mask;
        p.w = 0;
    }
}

// A table that one warp fills in insertion order, 32 elements at a time: a word per slot, (number << 18 | column) or kFree.  Lanes claim
// their slots by an atomic minimum and look who has them; those that lost go on, all at once.  Few rounds do (2.5 to 5 per batch
// for sets from power-law matrices, whatever the length of the table), and there is no chain of elements that push one another
// on.  Elements of later batches come after all that is in the table: a bit per slot says what is taken, and a lane reads the ten
// bits of its window and has its first free slot.  (A match of the lanes' slots in place of the claims holds the warp for some 230 cycles: twice
// the time.  The first batch, which is all of most sets, through the bits as well: 258 us for 31 k sets of up to 76 columns, now 196.)
struct BitTable {
    static constexpr int kShift = 18;
    SharedWords words, bits;
    __device__ __forceinline__ static unsigned column_of(unsigned w) { return w & ((1u << kShift) - 1u); }
    // The first n columns of the list into the table, emptied to `size` slots, and back to the list in slot order.
    template <class List>
    __device__ __forceinline__ void reorder(const List& list, int n, int size) const {
        const unsigned mask = (unsigned)size - 1u;
        const int lane = threadIdx.x & 31;
        for (int w = lane * 4; w < size; w += 128) words.free4(w);
        {
            const bool in = lane < n;
            const unsigned column = in ? list.ld(lane) : 0u, me = (unsigned)lane << kShift | column;
            Probe p = probe_begin(column, mask);
            __syncwarp();
            if (in) words.claim(p.i, me);
            for (;;) {
                __syncwarp();
                const bool lost = in && words.ld(p.i + p.w) != me;
                if (!__any_sync(0xffffffffu, lost)) break;
                if (lost) {
                    probe_advance(p, mask);
                    words.claim(p.i + p.w, me);
                }
            }
            if (n > 32) {
                for (int w = lane; w <= size >> 5; w += 32) bits.st(w, 0u);
                __syncwarp();
                bits.set((p.i + p.w) >> 5, 1u << ((p.i + p.w) & 31u));
                __syncwarp();
            }
        }
        for (int q0 = 32; q0 < n; q0 += 32) {
            const bool in = q0 + lane < n;
            const unsigned column = in ? list.ld(q0 + lane) : 0u, me = (unsigned)(q0 + lane) << kShift | column;
            Probe p = probe_begin(column, mask);
            if (in) {
                to_free(bits, p, mask);
                words.claim(p.i + p.w, me);
            }
            for (;;) {
                __syncwarp();
                const bool lost = in && words.ld(p.i + p.w) != me;
                if (!__any_sync(0xffffffffu, lost)) break;
                if (lost) {
                    ++p.w;
                    to_free(bits, p, mask);
                    words.claim(p.i + p.w, me);
                }
            }
            if (in) bits.set((p.i + p.w) >> 5, 1u << ((p.i + p.w) & 31u));
            __syncwarp();
        }
        int done = 0;
#pragma unroll 4
        for (int s0 = 0; s0 < size; s0 += 32) {
            const unsigned w = s0 + lane < size ? words.ld(s0 + lane) : kFree;
            const unsigned taken = __ballot_sync(0xffffffffu, w != kFree);
            if (w != kFree) list.st(done + __popc(taken & ((1u << lane) - 1u)), column_of(w));
            done += __popc(taken);
        }
        __syncwarp();
    }
    // Slot of a column; false: it is not in the table.
    __device__ __forceinline__ bool find(unsigned mask, unsigned column, unsigned& slot) const {
        Probe p = probe_begin(column, mask);
        for (unsigned n = 0; n <= 8u * mask + 64u; ++n) {
            slot = p.i + p.w;
            const unsigned w = words.ld(slot);
            if (w == kFree) return false;
            if (column_of(w) == column) return true;
            probe_advance(p, mask);
        }
        return false;
    }
    // The bits of the whole table, and in counts how many slots are taken before each word of them; then rank is a slot's place in the order.
    __device__ __forceinline__ void index(const SharedWords& counts, int size) const {
        const int lane = threadIdx.x & 31;
        int done = 0;
        for (int s0 = 0; s0 < size; s0 += 32) {
            const unsigned taken = __ballot_sync(0xffffffffu, s0 + lane < size && words.ld(s0 + lane) != kFree);
            if (lane == 0) {
                bits.st(s0 >> 5, taken);
                counts.st(s0 >> 5, (unsigned)done);
            }
            done += __popc(taken);
        }
        __syncwarp();
    }
    __device__ __forceinline__ int rank(const SharedWords& counts, unsigned slot) const {
        return (int)counts.ld(slot >> 5) + __popc(bits.ld(slot >> 5) & ((1u << (slot & 31u)) - 1u));
    }
};

constexpr int kWarpLevels = 128;      // CTA teams: tables up to this length are done by one warp
constexpr int kWarpLevelBits = 8;     // words of their bits (five are in use)
// Longer tables, up to this length, are filled in batches by teams of up to 512 threads, and are empty at the start of every level; the others
// are kept from one rebuild to the next.  Rows of neighbours take as many rounds as they are long, which a CTA of 1024 pays for most: stack of 16
// (V = 8), classes M1 and M2 394 and 487 us with kept tables, 263 and 453 so (12 matrices, V = 16: 502 and 937, 527 and 701), class L 578
// with kept tables, 1110 with batches up to 2048 slots, 1772 at all lengths.
constexpr int kBatchLevels = 2048;

// A set being rebuilt.  `list` is the insertion sequence: what the set held, in its order, then the row's new columns; a level's
// extraction writes the order of its table over the part that the level inserted.  A slot's word is the number of its
// element in the list and, packed (SHIFT bits), its column; unpacked the column is looked up in the list.  After the last level
// of the last rebuild the number is the position in the ordered set, so a word also answers where a column went.
// Tables up to BATCH slots are empty at the start of a level.  Packed, every longer level has a table of its own behind them, which
// stays for the next rebuild: between two rebuilds its words have the number kVacant (later than every element's), which a new element takes
// like a free slot.
enum class After { kFreed, kVacated, kNumbered };     // what becomes of a level's words when its order has been read
template <class Words, class List, int SHIFT, int BATCH>
struct HashSet {
    Words tab;
    List list;
    SharedWords bits;         // of the table of a batch level
    GlobalWords ext;          // unpacked only: extraction goes here first, since words refer to the list
    static constexpr bool kPacked = SHIFT > 0;
    static constexpr int kBatch = BATCH;
    static constexpr unsigned kVacant = kPacked ? ((1u << (32 - SHIFT)) - 2u) << SHIFT : kFree;      // words from here on name no element
    // where the table of a level starts (lengths grow by four as long as words are packed)
    __device__ __forceinline__ static unsigned start(int size) { return kPacked && size > BATCH ? (unsigned)(BATCH + (size - 4 * BATCH) / 3) : 0u; }
    __device__ __forceinline__ HashSet level(int size) const { return HashSet{tab.part(start(size)), list, bits, ext}; }
    __device__ __forceinline__ unsigned word(unsigned number, unsigned key) const { return kPacked ? number << SHIFT | key : number; }
    __device__ __forceinline__ unsigned key_of(unsigned w) const { return kPacked ? w & ((1u << SHIFT) - 1u) : list.ld(w); }
    __device__ __forceinline__ static unsigned number_of(unsigned w) { return w >> SHIFT; }
    // slot of a column, or of the free slot at which its path ends (the loop is bounded; a table is never more than 60 % full)
    __device__ __forceinline__ unsigned find(unsigned mask, unsigned key, unsigned& word) const {
        Probe p = probe_begin(key, mask);
        word = kFree;
        for (unsigned n = 0; n <= 8u * mask + 64u; ++n) {
            word = tab.ld(p.i + p.w);
            if (word == kFree || key_of(word) == key) break;
            probe_advance(p, mask);
        }
        return p.i + p.w;
    }
    __device__ __forceinline__ bool contains(unsigned mask, unsigned key) const {
        unsigned w;
        find(mask, key, w);
        return w != kFree;
    }
    // Insertion is first come, first served: an element takes a slot by an atomic minimum; whoever loses one (the element
    // itself, or a later one that had come to sit there) goes on along its path from there.  In a table that was free before, slots
    // only ever get earlier owners, so what was lost stays lost and the result does not depend on timing.
    // walk: from path position p on, until a slot was free.  True: a column occurs twice (or a bound was hit).
    __device__ __forceinline__ bool walk(unsigned me, unsigned mine, Probe p, unsigned mask) const {
        for (unsigned steps = 0; steps <= 64u * mask + 4096u; ++steps) {
            const unsigned slot = p.i + p.w;
            const unsigned cur = tab.take(slot, me);
            if (cur >= kVacant) return false;
            const unsigned other = key_of(cur);
            if (other == mine) return true;
            if (cur > me) {
                me = cur;
                mine = other;
                p = probe_at(mine, mask, slot);
            }
            probe_advance(p, mask);
        }
        return true;
    }
    // Elements first, first + stride, ... below n into a free table.  All are first tried at their home slots, four at a time and
    // without a branch; only losers walk.
    __device__ __forceinline__ bool insert(int n, unsigned mask, int first, int stride) const {
        constexpr int kTry = 4;
        for (int q0 = first; q0 < n; q0 += kTry * stride) {
            unsigned key[kTry], old[kTry];
#pragma unroll
            for (int b = 0; b < kTry; ++b) key[b] = q0 + b * stride < n ? list.ld(q0 + b * stride) : 0u;
#pragma unroll
            for (int b = 0; b < kTry; ++b)
                old[b] = q0 + b * stride < n ? tab.take(key[b] & mask, word(q0 + b * stride, key[b])) : kFree;
            bool again = false;
            unsigned lost[kTry];
            int losers = 0;
#pragma unroll
            for (int b = 0; b < kTry; ++b)
                if (old[b] < kVacant) {
                    again |= key_of(old[b]) == key[b];
#pragma unroll
                    for (int x = kTry - 1; x > 0; --x) lost[x] = lost[x - 1];
                    lost[0] = max(old[b], word(q0 + b * stride, key[b]));
                    ++losers;
                }
            bool walking = false;
            unsigned me = 0, mine = 0, steps = 0;
            Probe p = probe_begin(0, mask);
            while (!again && (walking || losers > 0)) {
                if (!walking) {                                   // the next loser; its home slot is out of reach
                    me = lost[0];
                    mine = key_of(me);
#pragma unroll
                    for (int x = 0; x + 1 < kTry; ++x) lost[x] = lost[x + 1];
                    --losers;
                    p = probe_begin(mine, mask);
                    probe_advance(p, mask);
                    walking = true;
                }
                const unsigned slot = p.i + p.w;
                const unsigned cur = tab.take(slot, me);
                if (cur >= kVacant) {
                    walking = false;
                } else {
                    const unsigned other = key_of(cur);
                    again = other == mine;
                    if (cur > me) {
                        me = cur;
                        mine = other;
                        p = probe_at(mine, mask, slot);
                    }
                    probe_advance(p, mask);
                    again |= ++steps > 64u * mask + 4096u;
                }
            }
            if (again) return true;
        }
        return false;
    }
    // The first n elements into an empty table, as BitTable's batches, of one element per thread.  A round is a barrier: whoever lost its
    // slot goes on and claims the next one, and when nobody has, all are in place.  (insert and relevel walk the losers one link after
    // another, on one thread each.)
    template <class Team>
    __device__ __forceinline__ void insert_batches(int n, int size) const {
        const unsigned mask = (unsigned)size - 1u;
        for (int w = threadIdx.x; w <= size >> 5; w += Team::kSize) bits.st(w, 0u);
        for (int q0 = 0; q0 < n; q0 += Team::kSize) {
            const bool in = q0 + (int)threadIdx.x < n;
            const unsigned key = in ? list.ld(q0 + threadIdx.x) : 0u, me = word(q0 + threadIdx.x, key);
            Probe p = probe_begin(key, mask);
            if (in) {
                if (q0 > 0) to_free(bits, p, mask);
                tab.claim(p.i + p.w, me);
            }
            bool lost = in;
            while (Team::any(lost, nullptr)) {
                lost = in && tab.ld(p.i + p.w) != me;
                if (lost) {
                    if (q0 > 0) {
                        ++p.w;
                        to_free(bits, p, mask);
                    } else {
                        probe_advance(p, mask);
                    }
                    tab.claim(p.i + p.w, me);
                }
            }
            if (in) bits.set((p.i + p.w) >> 5, 1u << ((p.i + p.w) & 31u));
            Team::sync();
        }
    }
    // Whether every slot on the path of the element in `slot` before that one has an earlier element.
    __device__ __forceinline__ bool in_place(unsigned w, unsigned slot, unsigned mask) const {
        Probe p = probe_begin(key_of(w), mask);
        for (unsigned n = 0; p.i + p.w != slot && n <= 8u * mask + 64u; ++n) {
            if (tab.ld(p.i + p.w) > w) return false;
            probe_advance(p, mask);
        }
        return true;
    }
    // One warp: levels from length 8 up to `last`; the level of length `final` is kept, in this table's first slots, which are free otherwise.
    __device__ __forceinline__ void warp_levels(const BitTable& b, int n_total, int last, int final) const {
        const int lane = threadIdx.x & 31;
        for (int size = kMinTable; size <= last; size = level_next(size)) b.reorder(list, min(level_trigger(size), n_total), size);
        int done = 0;
        for (int s0 = 0; s0 < (final <= last ? final : 0); s0 += 32) {
            const unsigned w = s0 + lane < final ? b.words.ld(s0 + lane) : kFree;
            const unsigned taken = __ballot_sync(0xffffffffu, w != kFree);
            if (s0 + lane < final) tab.st(s0 + lane, w != kFree ? word(done + __popc(taken & ((1u << lane) - 1u)), BitTable::column_of(w)) : kFree);
            done += __popc(taken);
        }
        __syncwarp();
    }
};

// Sequential replay by one thread (a matrix row lists a column twice; rare).  The table holds columns until the end; the list is
// overwritten in place: when a growing table is emptied into its head, that part of the sequence has been inserted.
template <class Set>
__device__ int replay_sequential(const SvcProblem& p, const int* rows, int n_rows, const Set& t, int cap, unsigned& mask_out) {
    int n_cur = 0;
    unsigned mask = kMinTable - 1;
    auto slot_of = [&](unsigned m, unsigned key) {
        Probe pr = probe_begin(key, m);
        for (unsigned n = 0; n <= 8u * m + 64u; ++n) {
            const unsigned e = t.tab.ld(pr.i + pr.w);
            if (e == key || e == kFree) break;
            probe_advance(pr, m);
        }
        return pr.i + pr.w;
    };
    for (int r = 0; r < n_rows; ++r) {
        const int rs = rows[r], rlen = rows[r + 1] - rs;
        int size = kMinTable, used = 0;
        mask = kMinTable - 1;
        for (int s = 0; s < size; ++s) t.tab.st(s, kFree);
        for (int x = 0; x < n_cur + rlen; ++x) {
            const unsigned key = x < n_cur ? t.list.ld(x) : (unsigned)p.col_idx[rs + x - n_cur];
            if (key >= (unsigned)p.K) continue;
            const unsigned s = slot_of(mask, key);
            if (t.tab.ld(s) == key) continue;
            t.tab.st(s, key);
            if (++used >= level_trigger(size)) {
                const int next = min(level_next(size), cap);
                int cnt = 0;
                for (int q = 0; q < size; ++q) if (t.tab.ld(q) != kFree) t.list.st(cnt++, t.tab.ld(q));
                for (int q = 0; q < next; ++q) t.tab.st(q, kFree);
                mask = (unsigned)next - 1u;
                for (int q = 0; q < cnt; ++q) { const unsigned k = t.list.ld(q); t.tab.st(slot_of(mask, k), k); }
                size = next;
            }
        }
        n_cur = 0;
        for (int q = 0; q < size; ++q) if (t.tab.ld(q) != kFree) t.list.st(n_cur++, t.tab.ld(q));
    }
    int n = 0;
    for (unsigned s = 0; s <= mask; ++s)
        if (t.tab.ld(s) != kFree) { const unsigned key = t.tab.ld(s); t.tab.st(s, t.word(n++, key)); }
    mask_out = mask;
    return n_cur;
}

// CTA team: the table's columns in slot order to the list.  Every warp owns a run of rows of 32 slots.
template <class Team, class Set>
__device__ __forceinline__ void extract_cta(const Set& t, int size, After after, int* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows = max(1, size / Team::kSize);
    const int first = warp * rows * 32 + lane;
    const bool in = warp * rows * 32 < size;
    int cnt = 0;
    if (in && size <= Set::kBatch)
        cnt = warp_sum(lane < rows ? __popc(t.bits.ld(warp * rows + lane)) : 0);        // (at most eight rows of a warp)
    else if (in)
#pragma unroll 4
        for (int j = 0; j < rows; ++j) cnt += __popc(__ballot_sync(0xffffffffu, t.tab.ld(first + j * 32) < Set::kVacant));
    int total;
    int pos = Team::before(cnt, total, red);
    if (in)
        for (int j0 = 0; j0 < rows; j0 += 4) {
            unsigned w[4], key[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) w[b] = j0 + b < rows ? t.tab.ld(first + (j0 + b) * 32) : kFree;
#pragma unroll
            for (int b = 0; b < 4; ++b) key[b] = w[b] < Set::kVacant ? t.key_of(w[b]) : 0u;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const unsigned m = __ballot_sync(0xffffffffu, w[b] < Set::kVacant);
                if (w[b] < Set::kVacant) {
                    const int x = pos + __popc(m & ((1u << lane) - 1u));
                    if (Set::kPacked) t.list.st(x, key[b]); else t.ext.st(x, key[b]);
                    t.tab.st(first + (j0 + b) * 32, after == After::kNumbered ? t.word(x, key[b]) : after == After::kVacated ? Set::kVacant | key[b] : kFree);
                } else if (w[b] != kFree) {
                    t.tab.st(first + (j0 + b) * 32, kFree);         // an element that left this level
                }
                pos += __popc(m);
            }
        }
    Team::sync();
    if (!Set::kPacked) {
        for (int q = threadIdx.x; q < total; q += Team::kSize) t.list.st(q, t.ext.ld(q));
        Team::sync();
    }
}

// A level whose table still has the columns of the rebuild before, vacated.  Most elements end where they ended then (a row adds
// a few columns to the set, and few elements change their order), and inserting them one after another into a free table is what
// costs: an element that comes to sit in an earlier one's place is pushed on, pushes the next one, and so on, up to 200 links one
// after another for 18 k columns.  So elements start from their old slots, the others are inserted, and then every element is
// checked: the one assignment in which each element has the first slot of its path that no earlier element holds is the result
// of inserting them in turn, whatever it was reached from.  Elements that are not in place are inserted again, until
// all are (the first wrong one in insertion order is final after a round, so there is an end; few rounds do in practice).
// Links on the critical path, 33903 columns, one row of 17.8 k: 12243 over all rebuilds from free tables, of which 600 are left.
template <class Team, class Set>
__device__ __forceinline__ bool relevel(const Set& t, int n, int size, int* red) {
    const int tid = threadIdx.x;
    const unsigned mask = (unsigned)size - 1u;
    unsigned todo = 0;                                     // a bit per element of this thread: not in the table
    for (int k0 = 0; k0 * Team::kSize < n; k0 += 4) {
        unsigned key[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) key[b] = (k0 + b) * Team::kSize + tid < n ? t.list.ld((k0 + b) * Team::kSize + tid) : 0u;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int q = (k0 + b) * Team::kSize + tid;
            if (q >= n) break;
            unsigned w;
            const unsigned slot = t.find(mask, key[b], w);
            if (w == kFree) todo |= 1u << (k0 + b);
            else t.tab.st(slot, t.word(q, key[b]));        // same column: other searches see no difference
        }
    }
    Team::sync();
    bool again = false;
    for (; todo && !again; todo &= todo - 1u) {
        const int q = (__ffs(todo) - 1) * Team::kSize + tid;
        const unsigned key = t.list.ld(q);
        again = t.walk(t.word(q, key), key, probe_begin(key, mask), mask);
    }
    Team::sync();
    constexpr int kRounds = 64;
    for (int round = 0; round <= kRounds; ++round) {
        for (int j = 0; j * Team::kSize + tid < size; ++j) {
            const unsigned s = j * Team::kSize + tid, w = t.tab.ld(s);
            if (w < Set::kVacant && (t.key_of(w) & mask) != s && !t.in_place(w, s, mask)) todo |= 1u << j;
        }
        if (!Team::any(again || todo != 0, red)) return false;
        if (Team::any(again, red)) return true;
        for (; todo && !again; todo &= todo - 1u) {
            const unsigned s = (__ffs(todo) - 1) * Team::kSize + tid, w = t.tab.ld(s);
            // (not there any more: someone has pushed it on)
            if (w < Set::kVacant && t.tab.give_up(s, w)) again = t.walk(w, t.key_of(w), probe_begin(t.key_of(w), mask), mask);
        }
        todo = 0;
        Team::sync();
    }
    for (int s = tid * 4; s < size; s += Team::kSize * 4) t.tab.free4(s);
    Team::sync();
    return Team::any(t.insert(n, mask, tid, Team::kSize), red);
}

// One group, by a CTA.  rows: kRowInts ints of shared memory; red: 96; small: kWarpLevels + kWarpLevelBits words.
template <class Team, class Set>
__device__ void replay_group(const SvcProblem& p, int i, int u_final, int cap, int base, const Set& t, const SharedWords& small, int* rows, int* red,
                             int* __restrict__ out_col, __half* __restrict__ out_vals) {
    constexpr bool kKeep = Set::kPacked;
    const int tid = Team::tid(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = min(i * p.V, p.M), n_rows = min(i * p.V + p.V, p.M) - r0;
    if (tid <= n_rows) rows[tid] = p.row_ptr[r0 + tid];
    for (int s = tid * 4; s < (int)Set::start(cap) + cap; s += Team::kSize * 4) t.tab.free4(s);
    if (out_vals && p.zero_values) zero_values<Team>(out_vals, base, u_final, p.V);
    Team::sync();
    auto table = [&](int size) { return kKeep ? t.level(size) : t; };

    int n_cur = 0, size = 0;                   // length of the table of the last rebuild (0: none yet, all slots free)
    bool again = false;
    int turn = 0;                              // which of two sets of warp counts is in use
    int next_key = tid < rows[1] - rows[0] ? p.col_idx[rows[0] + tid] : -1;          // the next row's columns are under way early
    for (int r = 0; r < n_rows; ++r) {
        const int rs = rows[r], rlen = rows[r + 1] - rs;
        int key = next_key;
        if (r + 1 < n_rows) next_key = tid < rows[r + 2] - rows[r + 1] ? p.col_idx[rows[r + 1] + tid] : -1;
        // ---- columns of this row that are not in the set yet, in row order
        const Set held = table(size);
        int n_new = 0;
        bool ascending = true;
        for (int t0 = 0; t0 < rlen; t0 += Team::kSize) {
            const bool in = t0 + tid < rlen;
            if (t0 > 0) key = in ? p.col_idx[rs + t0 + tid] : -1;
            if (in && t0 + tid > 0) ascending = ascending && p.col_idx[rs + t0 + tid - 1] < key;
            const bool fresh = (unsigned)key < (unsigned)p.K && (n_cur == 0 || !held.contains((unsigned)size - 1u, (unsigned)key));
            const unsigned b = __ballot_sync(0xffffffffu, fresh);
            int at = n_cur + n_new + __popc(b & ((1u << lane) - 1u));
            int total;
            at += Team::before(__popc(b), total, red + 32 + 32 * turn);
            n_new += total;
            turn ^= 1;
            if (fresh && at < u_final) t.list.st(at, (unsigned)key);
        }
        const int n_total = n_cur + n_new;
        if (n_total > u_final) { again = true; break; }     // only possible when the row repeats a column
        if (n_total == 0) continue;
        int final = kMinTable;
        while (n_total >= level_trigger(final)) final = level_next(final);
        // ---- set(list), level by level
        const bool unsorted = Team::any(!ascending, red);   // (the barrier: the list is complete, the table has been read)
        const int used = Set::start(size) > 0 ? 0 : size;   // tables of their own stay
        if (warp == 0) {
            for (int s = lane * 4; s < min(used, kWarpLevels); s += 128) t.tab.free4(s);
            __syncwarp();
            t.warp_levels(BitTable{small, small.part(kWarpLevels)}, n_total, min(final, kWarpLevels), final);
        } else {
            for (int s = kWarpLevels + (tid - 32) * 4; s < used; s += (Team::kSize - 32) * 4) t.tab.free4(s);
        }
        Team::sync();
        for (int level = level_next(kWarpLevels); level <= final && !again; level = level_next(level)) {
            const int n = min(level_trigger(level), n_total);
            if (level <= Set::kBatch) {
                t.template insert_batches<Team>(n, level);
                extract_cta<Team>(t, level, level == final ? After::kNumbered : After::kFreed, red);
                continue;
            }
            const Set l = table(level);
            if (kKeep && level <= size) again = relevel<Team>(l, n, level, red);
            else again = Team::any(l.insert(n, (unsigned)level - 1u, tid, Team::kSize), red);
            if (!again)
                extract_cta<Team>(l, level, level == final && (!kKeep || r + 1 == n_rows) ? After::kNumbered : kKeep ? After::kVacated : After::kFreed, red);
        }
        // A column that a row repeats is met in the tables above BATCH; in the others it has two slots, and only the first is found.
        if (unsorted && final <= Set::kBatch) {
            const Set now = table(final);
            bool twice = false;
            for (int q = tid; q < n_total; q += Team::kSize) {
                unsigned w;
                now.find((unsigned)final - 1u, t.list.ld(q), w);
                twice = twice || w == kFree || Set::number_of(w) != (unsigned)q;
            }
            again = Team::any(twice, red);
        }
        if (again) break;
        n_cur = n_total;
        size = final;
    }
    if (again) {
        unsigned mask = 0;
        Team::sync();
        if (tid == 0) { n_cur = replay_sequential(p, rows, n_rows, table(cap), cap, mask); size = (int)mask + 1; }
        n_cur = Team::broadcast(n_cur, red);
        size = Team::broadcast(size, red);
    }
    // the list is the ordered set, the words of the table name positions in it
    const Set held = table(size);
    for (int q = tid; q < n_cur; q += Team::kSize) out_col[base + q] = (int)t.list.ld(q);
    if (out_vals)
        for_each_value<Team>(p, rows, n_rows, [&](int r, int c, __half v) {
            unsigned w;
            held.find((unsigned)size - 1u, (unsigned)c, w);
            if (w != kFree) out_vals[((int64_t)base + Set::number_of(w)) * p.V + r] = v;
        });
    Team::sync();
}

// One group, by a warp.  What bounds it is the issue of instructions: 30 to 48 warps per SM, a few hundred instructions per rebuild.
// counts: a word per word of the table's bits.
__device__ void replay_group_by_warp(const SvcProblem& p, int i, int u_final, int cap, int base, const BitTable& t, const SharedWords& list,
                                     const SharedWords& counts, int* rows, int* __restrict__ out_col, __half* __restrict__ out_vals) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int r0 = min(i * p.V, p.M), n_rows = min(i * p.V + p.V, p.M) - r0;
    if (lane <= n_rows) rows[lane] = p.row_ptr[r0 + lane];
    if (out_vals && p.zero_values) zero_values<WarpTeam>(out_vals, base, u_final, p.V);
    __syncwarp();
    int n_cur = 0, size = kMinTable;
    bool again = false;
    int next_key = lane < rows[1] - rows[0] ? p.col_idx[rows[0] + lane] : -1;          // the next row's columns are under way early
    for (int r = 0; r < n_rows; ++r) {
        const int rs = rows[r], rlen = rows[r + 1] - rs;
        int key = next_key;
        if (r + 1 < n_rows) next_key = lane < rows[r + 2] - rows[r + 1] ? p.col_idx[rows[r + 1] + lane] : -1;
        // ---- columns of this row that are not in the set yet, in row order
        int n_total = n_cur, last = -1;
        bool ascending = true;
        for (int t0 = 0; t0 < rlen; t0 += 32) {
            const bool in = t0 + lane < rlen;
            if (t0 > 0) key = in ? p.col_idx[rs + t0 + lane] : -1;
            const int left = __shfl_up_sync(0xffffffffu, key, 1);
            ascending = ascending && (!in || (lane > 0 ? left : last) < key);
            last = __shfl_sync(0xffffffffu, key, 31);
            unsigned slot;
            const bool fresh = (unsigned)key < (unsigned)p.K && (n_cur == 0 || !t.find((unsigned)size - 1u, (unsigned)key, slot));
            const unsigned b = __ballot_sync(0xffffffffu, fresh);
            const int at = n_total + __popc(b & below);
            if (fresh && at < u_final) list.st(at, (unsigned)key);
            n_total += __popc(b);
        }
        if (n_total > u_final) { again = true; break; }     // only possible when the row repeats a column
        if (n_total == 0) continue;
        int final = kMinTable;
        while (n_total >= level_trigger(final)) final = level_next(final);
        __syncwarp();
        for (int level = kMinTable; level <= final; level = level_next(level)) t.reorder(list, min(level_trigger(level), n_total), level);
        n_cur = n_total;
        size = final;
        // a column that occurs twice has two slots now, and only the first of them is found
        if (!__all_sync(0xffffffffu, ascending)) {
            t.index(counts, size);
            for (int q0 = 0; q0 < n_cur && !again; q0 += 32) {
                unsigned slot = 0;
                const bool twice = q0 + lane < n_cur && (!t.find((unsigned)size - 1u, list.ld(q0 + lane), slot) || t.rank(counts, slot) != q0 + lane);
                again = __any_sync(0xffffffffu, twice);
            }
        }
        if (again) break;
    }
    if (again) {
        unsigned mask = 0;
        __syncwarp();
        if (lane == 0) n_cur = replay_sequential(p, rows, n_rows, HashSet<SharedWords, SharedWords, BitTable::kShift, kWarpLevels>{t.words, list, t.bits, GlobalWords{nullptr}}, cap, mask);
        n_cur = __shfl_sync(0xffffffffu, n_cur, 0);
        size = (int)__shfl_sync(0xffffffffu, mask, 0) + 1;
        __syncwarp();
    }
    for (int q = lane; q < n_cur; q += 32) out_col[base + q] = (int)list.ld(q);
    if (out_vals && n_cur > 0) {
        t.index(counts, size);
        for_each_value<WarpTeam>(p, rows, n_rows, [&](int r, int c, __half v) {
            unsigned slot;
            if (t.find((unsigned)size - 1u, (unsigned)c, slot)) out_vals[((int64_t)base + t.rank(counts, slot)) * p.V + r] = v;
        });
    }
    __syncwarp();
}

// What a team of a class has in shared memory: its tables, a list and the row ends of its group.  Class L with a table per level
// leaves no room for the list, and class XL has everything, in global scratch.
// SHIFT: bits of a column in a word; numbers of a list and two more fit the others (0: unpacked).
template <int CLASS, int SHIFT>
struct ClassShape {
    static constexpr bool kWarp = CLASS == kClassXS || CLASS == kClassS;
    static constexpr int kTeam = kWarp ? 32 : CLASS == kClassM1 ? 256 : CLASS == kClassM2 ? 512 : 1024;
    static constexpr int kCapU = CLASS == kClassXS ? kXSCapU : CLASS == kClassS ? kSCapU : CLASS == kClassM1 ? kM1CapU : CLASS == kClassM2 ? kM2CapU : kLCapU;
    static constexpr int kCapT = CLASS == kClassXS ? kXSCapT : CLASS == kClassS ? kSCapT : CLASS == kClassM1 ? kM1CapT : CLASS == kClassM2 ? kM2CapT : kLCapT;
    static constexpr bool kListInSmem = CLASS != kClassXL && !(CLASS == kClassL && SHIFT > 0);
    static constexpr int kBatch = kTeam <= 512 ? kBatchLevels : kWarpLevels;       // a CTA: tables filled in batches
    static constexpr int kTable = CLASS == kClassXL ? 0 : !kWarp && SHIFT > 0 && kCapT > kBatch ? kCapT + kBatch + (kCapT - 4 * kBatch) / 3 : kCapT;
    static constexpr int kList = kListInSmem ? (kCapU + 3) & ~3 : 0;
    static constexpr int kBits = (kWarp ? kCapT : kBatch) / 32 + 4;         // (the word after the last is read)
    static constexpr int kCounts = kWarp ? kCapT / 32 : kWarpLevels + kWarpLevelBits;      // a CTA: the table of the small levels
    static constexpr int kInts = kTable + kList + kBits + kCounts + kRowInts;     // of a team, in shared memory
    static constexpr int kThreads = kWarp ? 256 : kTeam;          // of a block
    static constexpr int kBlocks = (kTeam == 1024 ? 1024 : 1536) / kThreads;      // per SM
    using Team = std::conditional_t<kWarp, WarpTeam, BlockTeam<kTeam>>;
    static constexpr int kPerBlock = kThreads / kTeam;
    using Words = std::conditional_t<CLASS == kClassXL, GlobalWords, SharedWords>;
    using List = std::conditional_t<kListInSmem, SharedWords, GlobalList>;
    static_assert(SHIFT == 0 || kCapU < (1ll << (32 - SHIFT)) - 2, "numbers of a list fit the words");
    static_assert(kWarp || SHIFT == 0 || (kCapU <= 32 * kTeam && kCapT <= 32 * kTeam), "relevel: a bit per element and slot of a thread");
};

template <int CLASS, int SHIFT>
__global__ void __launch_bounds__(ClassShape<CLASS, SHIFT>::kThreads, ClassShape<CLASS, SHIFT>::kBlocks)
svc_emit_replay_kernel(SvcProblem p, const int* __restrict__ vec_ptr, const int* __restrict__ tbl_len,
                       const long long* __restrict__ tbl_off, int* __restrict__ scratch, int* __restrict__ out_col,
                       __half* __restrict__ out_vals, const int* __restrict__ groups, int n_groups, int* __restrict__ queue) {
    using Shape = ClassShape<CLASS, SHIFT>;
    using Team = typename Shape::Team;
    static_assert(Shape::kInts % 4 == 0, "tables start on 16-byte boundaries");
    extern __shared__ __align__(16) int sm_ints[];
    __shared__ int red[96];
    int* mine = sm_ints + (size_t)Team::index_in_block() * Shape::kInts;
    const SharedWords bits{smem_u32(mine + Shape::kTable + Shape::kList)};
    int* const rows = mine + Shape::kTable + Shape::kList + Shape::kBits + Shape::kCounts;
    for (;;) {
        int k = 0;
        if (Team::tid() == 0) k = atomicAdd(queue, 1);
        k = Team::broadcast(k, red);
        if (k >= n_groups) break;
        const int i = groups[k];
        const int base = vec_ptr[i];
        const int u = vec_ptr[i + 1] - base;
        const int cap = tbl_len[i];
        if constexpr (Shape::kWarp) {
            replay_group_by_warp(p, i, u, cap, base, BitTable{SharedWords{smem_u32(mine)}, bits}, SharedWords{smem_u32(mine + Shape::kTable)},
                                 bits.part(Shape::kBits), rows, out_col, out_vals);
        } else {
            unsigned* g = reinterpret_cast<unsigned*>(scratch) + (CLASS == kClassL || CLASS == kClassXL ? tbl_off[i] : 0);
            HashSet<typename Shape::Words, typename Shape::List, SHIFT, Shape::kBatch> t;
            if constexpr (CLASS == kClassXL) { t.tab.at = g; g += cap; }
            else t.tab.at = smem_u32(mine);
            if constexpr (Shape::kListInSmem) t.list.at = smem_u32(mine + Shape::kTable);
            else { t.list.at = g; g += u; }
            t.bits = bits;
            t.ext.at = g;
            replay_group<Team>(p, i, u, cap, base, t, bits.part(Shape::kBits), rows, red, out_col, out_vals);
        }
    }
}

int device_sm_count() { return current_device_sm_count(); }

// Side streams so that launches working on disjoint groups overlap (fork from / join into the caller's stream).
constexpr int kAuxStreams = 6;
struct Aux {
    cudaStream_t stream[kAuxStreams];
    cudaEvent_t fork, join[kAuxStreams];
    bool ready = false;
};
std::mutex g_aux_mu;                 // serialises enqueueing through the shared events
Aux g_aux[64];

Aux* aux_for_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    Aux& a = g_aux[dev];
    if (!a.ready) {
        for (int k = 0; k < kAuxStreams; ++k) {
            if (cudaStreamCreateWithFlags(&a.stream[k], cudaStreamNonBlocking) != cudaSuccess) return nullptr;
            if (cudaEventCreateWithFlags(&a.join[k], cudaEventDisableTiming) != cudaSuccess) return nullptr;
        }
        if (cudaEventCreateWithFlags(&a.fork, cudaEventDisableTiming) != cudaSuccess) return nullptr;
        a.ready = true;
    }
    return &a;
}

struct Fork {
    Aux* aux;
    cudaStream_t main;
    int used = 0;
    cudaError_t err = cudaSuccess;
    Fork(Aux* a, cudaStream_t m) : aux(a), main(m) {
        if (aux) err = cudaEventRecord(aux->fork, main);
    }
    // stream for the next independent launch (the caller's stream when side streams are unavailable)
    cudaStream_t next() {
        if (!aux || used >= kAuxStreams || err != cudaSuccess) return main;
        cudaStream_t s = aux->stream[used++];
        err = cudaStreamWaitEvent(s, aux->fork, 0);
        return err == cudaSuccess ? s : main;
    }
    cudaError_t join() {
        if (!aux) return err;
        for (int k = 0; k < used && err == cudaSuccess; ++k) {
            err = cudaEventRecord(aux->join[k], aux->stream[k]);
            if (err == cudaSuccess) err = cudaStreamWaitEvent(main, aux->join[k], 0);
        }
        return err;
    }
};

template <int CLASS, int SHIFT>
cudaError_t launch_replay(const SvcProblem& p, const SvcScratch& s, int* out_col, __half* out_vals, long long groups,
                          long long first, cudaStream_t stream) {
    if (groups <= 0) return cudaSuccess;
    using Shape = ClassShape<CLASS, SHIFT>;
    auto kern = svc_emit_replay_kernel<CLASS, SHIFT>;
    const size_t smem = (size_t)Shape::kPerBlock * Shape::kInts * sizeof(int);
    static DeviceOnce once;
    if (!once.done()) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        // without this the driver may size the shared-memory carve-out for a single resident block
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        once.mark();
    }
    // as many blocks as can be resident: the groups are handed out through the class's work counter
    const long long want = (groups + Shape::kPerBlock - 1) / Shape::kPerBlock;
    const long long most = (long long)device_sm_count() * Shape::kBlocks;
    kern<<<(unsigned)(want < most ? want : most), Shape::kThreads, smem, stream>>>(p, s.vec_ptr, s.tbl_len, s.tbl_off, s.tables, out_col, out_vals,
                                                                            s.class_list + first, (int)groups, s.queue + CLASS);
    return cudaGetLastError();
}

template <class Kern>
cudaError_t allow_big_smem(Kern kern, DeviceOnce& once, int bytes) {
    if (once.done()) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) once.mark();
    return e;
}

}  // namespace

cudaError_t svc_count_and_scan(const SvcProblem& p, const SvcScratch& s, bool /*with_values*/, cudaStream_t stream) {
    if (p.m_vec > 0) {
        const int words = (p.K + 31) / 32;
        const int sms = device_sm_count();
        static DeviceOnce once_block, once_small, once_warp;
        cudaError_t e = allow_big_smem(svc_count_kernel<BlockTeam<kBigTeam>>, once_block, 200 * 1024);
        if (e == cudaSuccess) e = allow_big_smem(svc_count_kernel<BlockTeam<kTeam>>, once_small, 200 * 1024);
        if (e == cudaSuccess) e = allow_big_smem(svc_count_kernel<WarpTeam>, once_warp, 200 * 1024);
        if (e != cudaSuccess) return e;
        const size_t warp_smem = (size_t)WarpTeam::kPerBlock * words * 4;
        if (p.m_vec <= 16 * sms || warp_smem > 200 * 1024) {
            // few groups (or bitmaps too large for eight per block): one CTA per group
            const int grid = p.m_vec < sms * 16 ? p.m_vec : sms * 16;
            if (p.m_vec <= 2 * sms) svc_count_kernel<BlockTeam<kBigTeam>><<<grid, kBigTeam, (size_t)words * 4, stream>>>(p, words, 0, s.vec_ptr, s.mode, s.tbl_len);
            else svc_count_kernel<BlockTeam<kTeam>><<<grid, kTeam, (size_t)words * 4, stream>>>(p, words, 0, s.vec_ptr, s.mode, s.tbl_len);
            e = cudaGetLastError();
        } else {
            std::lock_guard<std::mutex> lk(g_aux_mu);
            Fork f(aux_for_device(), stream);
            int grid = (p.m_vec + WarpTeam::kPerBlock - 1) / WarpTeam::kPerBlock;
            if (grid > sms * 8) grid = sms * 8;
            svc_count_kernel<WarpTeam><<<grid, 256, warp_smem, f.next()>>>(p, words, 1, s.vec_ptr, s.mode, s.tbl_len);
            svc_count_kernel<BlockTeam<kBigTeam>><<<sms * 2, kBigTeam, (size_t)words * 4, f.next()>>>(p, words, 2, s.vec_ptr, s.mode, s.tbl_len);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = f.join();
        }
        if (e != cudaSuccess) return e;
    }
    const int n_blocks = p.m_vec > 0 ? (p.m_vec + kScanBlock - 1) / kScanBlock : 1;
    if (n_blocks == 1) {
        svc_scan_place_kernel<true><<<1, kScanThreads, 0, stream>>>(p.m_vec, s.vec_ptr, s.tbl_len, s.tbl_off, nullptr, s.totals, s.host_totals, s.class_list);
        return cudaGetLastError();
    }
    svc_scan_sums_kernel<<<n_blocks, kScanThreads, 0, stream>>>(p.m_vec, s.vec_ptr, s.tbl_len, s.block_sums);
    svc_scan_blocks_kernel<<<1, 32 * kScanFields, 0, stream>>>(n_blocks, s.block_sums, s.totals, s.host_totals);
    svc_scan_place_kernel<false><<<n_blocks, kScanThreads, 0, stream>>>(p.m_vec, s.vec_ptr, s.tbl_len, s.tbl_off, s.block_sums, s.totals, nullptr,
                                                                 s.class_list);
    return cudaGetLastError();
}

cudaError_t svc_emit(const SvcProblem& p, const SvcScratch& s, const long long* seg_groups, int* out_ptr, int* out_col,
                     __half* out_vals, cudaStream_t stream) {
    if (p.m_vec == 0) return cudaSuccess;
    const int sms = device_sm_count();
    const int words = (p.K + 31) / 32;
    static DeviceOnce once_block, once_small, once_warp;
    cudaError_t e = allow_big_smem(svc_emit_sorted_kernel<BlockTeam<kBigTeam>>, once_block, 208 * 1024);
    if (e == cudaSuccess) e = allow_big_smem(svc_emit_sorted_kernel<BlockTeam<kTeam>>, once_small, 208 * 1024);
    if (e == cudaSuccess) e = allow_big_smem(svc_emit_sorted_kernel<WarpTeam>, once_warp, 208 * 1024);
    if (e != cudaSuccess) return e;

    // groups per class and where the class starts in the list of replayed groups
    long long class_groups[kNumClasses] = {0}, first[kNumClasses] = {0};
    class_groups[kClassSorted] = seg_groups[0] + seg_groups[kSegSortedBig];
    long long big_first = 0;                       // the ascending groups that may need a CTA: last segment of the list
    for (int k = 1; k < kSegSortedBig; ++k) big_first += seg_groups[k];
    const int* big_list = s.class_list + big_first;
    const int n_big = (int)seg_groups[kSegSortedBig];
    for (int c = 1; c < kNumClasses; ++c) {
        int s0, s1;
        class_segments(c, s0, s1);
        for (int k = 1; k < s0; ++k) first[c] += seg_groups[k];
        for (int k = s0; k < s1; ++k) class_groups[c] += seg_groups[k];
    }
    long long replayed = 0;
    for (int c = 1; c < kNumClasses; ++c) replayed += class_groups[c];
    // the work counters of the replay classes, cleared before the side streams fork off
    if (replayed > 0) {
        e = cudaMemsetAsync(s.queue, 0, 8 * sizeof(int), stream);
        if (e != cudaSuccess) return e;
    }
    // Side streams only for launches that there are: a record or a wait costs the caller half a microsecond and the device's front end
    // more (weights without replayed groups: 6 records and 10 waits around one launch).
    const bool one_cta_each = p.m_vec <= 16 * sms || (size_t)WarpTeam::kPerBlock * words * 8 > 200 * 1024;
    const bool forks = replayed > 0 || (n_big > 0 && !one_cta_each);
    std::unique_lock<std::mutex> lk(g_aux_mu, std::defer_lock);
    if (forks) lk.lock();
    Fork f(forks ? aux_for_device() : nullptr, stream);
    if (out_ptr && class_groups[kClassSorted] == 0) {
        e = cudaMemcpyAsync(out_ptr, s.vec_ptr, ((size_t)p.m_vec + 1) * 4, cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) return e;
    }
    if (class_groups[kClassSorted] > 0) {
        const size_t warp_smem = (size_t)WarpTeam::kPerBlock * words * 8;
        if (one_cta_each) {
            const int grid = p.m_vec < sms * 16 ? p.m_vec : sms * 16;
            if (p.m_vec <= 2 * sms) svc_emit_sorted_kernel<BlockTeam<kBigTeam>><<<grid, kBigTeam, (size_t)words * 8, stream>>>(p, words, 0, s.vec_ptr, s.mode, out_ptr, out_col, out_vals, nullptr, 0);
            else svc_emit_sorted_kernel<BlockTeam<kTeam>><<<grid, kTeam, (size_t)words * 8, stream>>>(p, words, 0, s.vec_ptr, s.mode, out_ptr, out_col, out_vals, nullptr, 0);
        } else {
            int grid = (p.m_vec + WarpTeam::kPerBlock - 1) / WarpTeam::kPerBlock;
            if (grid > sms * 8) grid = sms * 8;
            svc_emit_sorted_kernel<WarpTeam><<<grid, 256, warp_smem, stream>>>(p, words, 1, s.vec_ptr, s.mode, out_ptr, out_col, out_vals, nullptr, 0);
            if (n_big > 0) {
                const int big_grid = n_big < sms * 2 ? n_big : sms * 2;
                svc_emit_sorted_kernel<BlockTeam<kBigTeam>><<<big_grid, kBigTeam, (size_t)words * 8, f.next()>>>(p, words, 2, s.vec_ptr, s.mode, nullptr, out_col,
                                                                                                     out_vals, big_list, n_big);
            }
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    // the largest groups first: they are the critical path
    auto replay = [&](auto kernel, int c, bool aside) {
        if (e == cudaSuccess && class_groups[c] > 0) e = kernel(p, s, out_col, out_vals, class_groups[c], first[c], aside ? f.next() : stream);
    };
    replay(launch_replay<kClassXL, 0>, kClassXL, true);
    replay(p.K <= 1 << 17 ? launch_replay<kClassL, 17> : launch_replay<kClassL, 0>, kClassL, true);
    replay(launch_replay<kClassM2, 18>, kClassM2, true);
    replay(launch_replay<kClassM1, 18>, kClassM1, true);
    replay(launch_replay<kClassS, 18>, kClassS, true);
    replay(launch_replay<kClassXS, 18>, kClassXS, false);
    if (e != cudaSuccess) return e;
    return f.join();
}


// ---- batches -------------------------------------------------------------------------------
namespace {
// index of the matrix that owns position x, for a table whose `base` member is ascending
template <class F>
__device__ __forceinline__ int owner_of(long long x, int count, F base_of) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base_of(mid) <= x) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Bound by its copies (6 bytes per entry each way).  A CTA takes runs of kStackRun positions: it looks the matrix of a run's first
// position up in the table (in shared memory when it came with the launch) and the threads walk on from there, four loads of each array under way.  Stack of 16,
// 5.3 M entries: 19 us, 24 with a search in global memory for every entry.
constexpr int kStackRun = 1024;
struct SvcStackTable {
    SvcBatchEntry e[kSvcParamEntries + 1];
};
// in_params: the table is in `given`, and CTA 0 also writes it to d_tab; else it is in d_tab.
__global__ void __launch_bounds__(256)
svc_stack_kernel(const __grid_constant__ SvcStackTable given, bool in_params, SvcBatchEntry* __restrict__ d_tab, int count, long long rows,
                 long long entries, int* __restrict__ row_ptr, int* __restrict__ col_idx, __half* __restrict__ vals) {
    __shared__ SvcBatchEntry near[kSvcParamEntries + 1];
    const SvcBatchEntry* tab = d_tab;
    if (in_params) {
        constexpr int kWords = sizeof(SvcBatchEntry) / 4;
        for (int x = threadIdx.x; x < (count + 1) * kWords; x += 256) {
            const int v = reinterpret_cast<const int*>(given.e)[x];
            reinterpret_cast<int*>(near)[x] = v;
            if (blockIdx.x == 0) reinterpret_cast<int*>(d_tab)[x] = v;
        }
        __syncthreads();
        tab = near;
    }
    const long long step = (long long)gridDim.x * kStackRun;
    for (long long r0 = (long long)blockIdx.x * kStackRun; r0 <= rows; r0 += step) {
        int m = owner_of(r0, count, [&](int k) { return tab[k].row_base; });
#pragma unroll
        for (int b = 0; b < kStackRun / 256; ++b) {
            const long long r = r0 + b * 256 + threadIdx.x;
            if (r > rows) break;
            if (r == rows) { row_ptr[r] = (int)entries; break; }
            while (m + 1 < count && tab[m + 1].row_base <= r) ++m;
            const long long lr = r - tab[m].row_base;
            row_ptr[r] = (int)(tab[m].nnz_base + (lr < tab[m].M ? tab[m].row_ptr[lr] : tab[m].nnz));
        }
    }
    for (long long e0 = (long long)blockIdx.x * kStackRun; e0 < entries; e0 += step) {
        int m = owner_of(e0, count, [&](int k) { return tab[k].nnz_base; });
        int c[kStackRun / 256];
        __half v[kStackRun / 256];
#pragma unroll
        for (int b = 0; b < kStackRun / 256; ++b) {
            const long long e = e0 + b * 256 + threadIdx.x;
            if (e >= entries) break;
            while (m + 1 < count && tab[m + 1].nnz_base <= e) ++m;
            const long long le = e - tab[m].nnz_base;
            c[b] = __ldg(tab[m].col_idx + le);
            if (vals) v[b] = tab[m].vals[le];
        }
#pragma unroll
        for (int b = 0; b < kStackRun / 256; ++b) {
            const long long e = e0 + b * 256 + threadIdx.x;
            if (e >= entries) break;
            col_idx[e] = c[b];
            if (vals) vals[e] = v[b];
        }
    }
}

__global__ void svc_batch_cuts_kernel(const SvcBatchEntry* __restrict__ tab, int count, const int* __restrict__ vec_ptr,
                                      long long* __restrict__ cuts, long long* __restrict__ host_cuts) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > count) return;
    const long long v = vec_ptr[tab[m].vec_row_base];
    cuts[m] = v;
    if (host_cuts) host_cuts[m] = v;
}

__global__ void __launch_bounds__(256)
svc_batch_row_ptrs_kernel(const SvcBatchEntry* __restrict__ tab, int count, long long vec_rows, const int* __restrict__ vec_ptr,
                          const long long* __restrict__ cuts, int* __restrict__ out) {
    // output position x = (stacked vector row) + (matrix index): each matrix has one pointer more than vector rows
    const long long total = vec_rows + count;
    for (long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += (long long)gridDim.x * blockDim.x) {
        const int m = owner_of(x, count, [&](int k) { return tab[k].vec_row_base + k; });
        const long long lv = x - tab[m].vec_row_base - m;
        out[x] = (int)(vec_ptr[tab[m].vec_row_base + lv] - cuts[m]);
    }
}
}  // namespace

cudaError_t svc_stack(const SvcBatchEntry* tab, SvcBatchEntry* d_tab, int count, long long rows, long long entries, int* row_ptr,
                      int* col_idx, __half* vals, cudaStream_t stream) {
    const long long work = (rows + 1 > entries ? rows + 1 : entries);
    long long blocks = (work + kStackRun - 1) / kStackRun;
    const long long cap = (long long)device_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    static_assert(sizeof(SvcStackTable) <= 4000, "the table fits the parameters of a launch");
    SvcStackTable given;
    const bool in_params = count <= kSvcParamEntries;
    if (in_params) {
        for (int k = 0; k <= count; ++k) given.e[k] = tab[k];
    } else {
        cudaError_t e = cudaMemcpyAsync(d_tab, tab, ((size_t)count + 1) * sizeof(SvcBatchEntry), cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);          // `tab` is pageable memory of the caller
        if (e != cudaSuccess) return e;
    }
    svc_stack_kernel<<<(int)blocks, 256, 0, stream>>>(given, in_params, d_tab, count, rows, entries, row_ptr, col_idx, vals);
    return cudaGetLastError();
}

cudaError_t svc_batch_cuts(const SvcBatchEntry* tab, int count, const int* vec_ptr, long long* cuts, long long* host_cuts, cudaStream_t stream) {
    svc_batch_cuts_kernel<<<(count + 1 + 255) / 256, 256, 0, stream>>>(tab, count, vec_ptr, cuts, host_cuts);
    return cudaGetLastError();
}

cudaError_t svc_batch_row_ptrs(const SvcBatchEntry* tab, int count, long long vec_rows, const int* vec_ptr,
                               const long long* cuts, int* out, cudaStream_t stream) {
    long long blocks = (vec_rows + count + 255) / 256;
    const long long cap = (long long)device_sm_count() * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    svc_batch_row_ptrs_kernel<<<(int)blocks, 256, 0, stream>>>(tab, count, vec_rows, vec_ptr, cuts, out);
    return cudaGetLastError();
}

cudaError_t svc_read_and_clear_bad_column_flag(int* flag, cudaStream_t stream) {
    cudaError_t e = cudaMemcpyFromSymbolAsync(flag, g_svc_bad_column, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return e;
    if (*flag) {
        const int zero = 0;
        e = cudaMemcpyToSymbolAsync(g_svc_bad_column, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    }
    return e;
}

}  // namespace sspmm_b200
