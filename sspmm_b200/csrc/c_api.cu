// extern "C" entry points declared in include/sspmm_b200.h.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/sspmm_b200.h"
#include "launch.h"
#include "ptx.cuh"
#include "svc.cuh"

namespace sspmm_b200 {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
}

static std::atomic<int> g_kernel_choice{0};

static int fail(cudaError_t e, const char* what) {
    if (g_err[0] == 0) set_error("%s: %s", what, cudaGetErrorString(e));
    return (int)e;
}

// The stream-ordered allocator returns memory to the OS at every synchronisation unless told to
// keep some; scratch is requested per call, so let the pool keep up to 1 GiB (once per device).
static void keep_pool_memory() {
    static DeviceOnce once;
    if (once.done()) return;
    int dev = 0;
    cudaMemPool_t pool;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        unsigned long long cur = 0, want = 1ull << 30;
        if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &cur) == cudaSuccess && cur < want)
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &want);
    }
    once.mark();
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// nvec = row_offsets[m_vec] lives in device memory; the kernel choice needs it on
// the host.  It is read once per (pointer, m_vec, device) and remembered: weights
// are static across calls.  A stale entry can only make the choice of kernel
// suboptimal, never the result wrong (both kernels accept any operand).
struct NvecEntry { const int* ptr; int m_vec; int dev; long long nvec; };
static std::mutex g_nvec_mu;
static NvecEntry g_nvec_cache[64];
static int g_nvec_next = 0;

static long long lookup_nvec(const int* row_offsets, int m_vec, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lk(g_nvec_mu);
        for (const NvecEntry& e : g_nvec_cache)
            if (e.ptr == row_offsets && e.m_vec == m_vec && e.dev == dev) return e.nvec;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return -1;
    int h = 0;
    if (cudaMemcpyAsync(&h, row_offsets + m_vec, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    std::lock_guard<std::mutex> lk(g_nvec_mu);
    g_nvec_cache[g_nvec_next] = NvecEntry{row_offsets, m_vec, dev, h};
    g_nvec_next = (g_nvec_next + 1) % 64;
    return h;
}

// Modelled times (seconds) of the two kernels, fitted to a sweep of shapes (64 to 2048 rows, K 64 to 4608, N 8 to 8192,
// sparsity 0.5 to 0.98, both V) measured on B200 in graph replays.  Row-gather kernel: launch and one chain of look-ups,
// then 2 * nvec * N bytes of gathers at 8.3 TB/s.  Block kernel: two launches, the dense copy of A written and read, the
// longer of its K loop's latency and its dense flops, and a third launch when few tiles make it cut K.  The last term is
// what the host pays for the scratch and the extra launches.  At the crossing (512 x 512, sparsity 0.5, V = 8): N = 128
// 5.4 against 9.3 us, N = 1024 11.1 against 9.4 us.
static bool block_kernel_is_faster(long long nvec, const SpmmArgs& a) {
    const double n = (double)a.N * a.batch;
    const double mp = (double)a.m_vec * a.V;
    const int sms = current_device_sm_count() > 0 ? current_device_sm_count() : 148;
    const double t_rows = 3.7e-6 + 2.0 * (double)nvec * n / 8.3e12;
    const double depth = 1.0e-9 * a.K, flops = 2.0 * mp * a.K * n / 1.25e15;
    const bool cuts_k = a.K >= 512 && (mp + 127) / 128 * ((a.N + 255) / 256) * a.batch < sms;
    const double t_block = 6.0e-6 + (cuts_k ? 2.8e-6 : 0.0) + 4.0 * mp * a.K / 3.8e12 + (depth > flops ? depth : flops) + 1.5e-6;
    return t_block < t_rows;
}

// Whether the block kernel can take the call at all (rhs_ok: the dense operand lies on 16-byte boundaries; TMA reads whole batches
// with one stride).
static bool block_fits(const SpmmArgs& a, bool rhs_ok) {
    const int64_t oes = a.out_f16 ? 2 : 4;
    const bool out_ok = aligned16(a.out) && ((int64_t)a.n_out * oes) % 16 == 0;
    return rhs_ok && out_ok && (a.batch == 1 || (a.values_stride == 0 && a.rhs_stride == (int64_t)a.K * a.n_out && (a.out_stride * oes) % 16 == 0)) &&
           sspmm_block_scratch_bytes(a) <= ((size_t)2 << 30);
}

// Length-sorted scheduling order: rank by (length descending, row id ascending).
__global__ void __launch_bounds__(256)
row_swizzle_kernel(int m_vec, const int* __restrict__ row_offsets, int* __restrict__ row_indices) {
    __shared__ int tile_len[256];
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int my = (i < m_vec) ? row_offsets[i + 1] - row_offsets[i] : 0;
    int rank = 0;
    for (int base = 0; base < m_vec; base += 256) {
        const int k = base + threadIdx.x;
        tile_len[threadIdx.x] = (k < m_vec) ? row_offsets[k + 1] - row_offsets[k] : -1;
        __syncthreads();
        const int lim = min(256, m_vec - base);
        for (int t = 0; t < lim; ++t) {
            const int l = tile_len[t];
            rank += (l > my || (l == my && base + t < i)) ? 1 : 0;
        }
        __syncthreads();
    }
    if (i < m_vec) row_indices[rank] = i;
}

// The same order for many rows: the rank loop above compares every row with every other (7e10 comparisons at
// 262 144 rows), so beyond a few thousand rows the rows are sorted instead.  Key = (2^32 - 1 - length) in the high
// word, row id in the low word: all keys differ, ascending keys are the wanted order.  Bitonic network over the next
// power of two of keys in global memory (padding keys are all ones and end up last).
constexpr int kSwizzleRankLimit = 8192;
__global__ void __launch_bounds__(256)
swizzle_keys_kernel(int m_vec, long long padded, const int* __restrict__ row_offsets, unsigned long long* __restrict__ keys) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= padded) return;
    unsigned long long k = ~0ull;
    if (i < m_vec) {
        const unsigned len = (unsigned)max(0, row_offsets[i + 1] - row_offsets[i]);
        k = ((unsigned long long)(0xffffffffu - len) << 32) | (unsigned)i;
    }
    keys[i] = k;
}
__global__ void __launch_bounds__(256)
swizzle_bitonic_kernel(long long padded, long long j, long long k, unsigned long long* __restrict__ keys) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= padded) return;
    const long long partner = i ^ j;
    if (partner <= i) return;
    const unsigned long long a = keys[i], b = keys[partner];
    const bool ascending = (i & k) == 0;
    if ((a > b) == ascending) { keys[i] = b; keys[partner] = a; }
}
__global__ void __launch_bounds__(256)
swizzle_write_kernel(int m_vec, const unsigned long long* __restrict__ keys, int* __restrict__ row_indices) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < m_vec) row_indices[i] = (int)(keys[i] & 0xffffffffull);
}

// Wait-expiry self test: one thread waits on an mbarrier that nobody arrives at.  The bounded wait
// must give up after g_wait_cycle_limit cycles, record kStatusWaitSelfTest and let the kernel return.
__global__ void wait_expiry_selftest_kernel(int* gave_up) {
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(smem_u32(&bar), 1);
        mbar_fence_init();
        const bool ok = mbar_wait(smem_u32(&bar), 0, &abort_flag, kStatusWaitSelfTest);
        *gave_up = ok ? 0 : 1;
    }
}

// Caller-provided knowledge and room: with nvec >= 0 nothing is read back from the device, with a workspace nothing
// is allocated.  query != null: only report the workspace size the chosen kernel wants, launch nothing.
struct SpmmExtra {
    long long nvec = -1;
    void* workspace = nullptr;
    size_t workspace_bytes = 0;
    bool caller_workspace = false;
    size_t* query = nullptr;
    const void* bias = nullptr;
};

static int spmm_entry(int m_vec, int V, int N, int K, int batch, const int* row_indices, const int* row_offsets,
                      const int* column_indices, const void* values, int64_t values_stride, const void* rhs,
                      int64_t rhs_stride, void* out, int64_t out_stride, bool out_f16, void* stream,
                      const SpmmExtra& ex = SpmmExtra()) {
    g_err[0] = 0;
    if (V != 8 && V != 16) {
        set_error("vec_length must be 8 or 16 (got %d)", V);
        return (int)cudaErrorInvalidValue;
    }
    if (m_vec < 0 || N < 0 || K < 0 || batch < 0) {
        set_error("negative dimension (m_vec=%d N=%d K=%d batch=%d)", m_vec, N, K, batch);
        return (int)cudaErrorInvalidValue;
    }
    if (ex.query) *ex.query = 0;
    if (m_vec == 0 || N == 0 || batch == 0) return 0;
    if (!ex.query && (!row_offsets || !out || (K > 0 && (!column_indices || !values || !rhs)))) {
        set_error("null operand pointer");
        return (int)cudaErrorInvalidValue;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    SpmmArgs a;
    a.m_vec = m_vec; a.V = V; a.N = N; a.n_out = N; a.K = K;
    a.row_indices = row_indices; a.row_offsets = row_offsets; a.column_indices = column_indices;
    a.values = static_cast<const __half*>(values); a.rhs = static_cast<const __half*>(rhs);
    a.out = out; a.out_f16 = out_f16; a.bias = static_cast<const __half*>(ex.bias); a.batch = batch;
    a.values_stride = values_stride; a.rhs_stride = rhs_stride; a.out_stride = out_stride;
    a.stream = st;

    int choice = g_kernel_choice.load();
    if (choice == 1 && a.bias) choice = 4;                     // the TMA gather kernel adds no bias
    const bool values_ok = aligned16(values) && (values_stride * 2) % 16 == 0;
    const bool rhs_ok = N % 8 == 0 && aligned16(rhs) && (batch == 1 || (rhs_stride * 2) % 16 == 0);
    if (choice == 1 && !(K > 0 && values_ok && rhs_ok && (batch == 1 || rhs_stride == (int64_t)K * N))) {
        set_error("tensor-core kernel needs N %% 8 == 0, 16-byte aligned values/rhs and contiguous batches");
        return (int)cudaErrorInvalidValue;
    }
    cudaError_t e;
    // The other kernels read 16-byte pieces.  A dense operand that does not lie on 16-byte boundaries (any N) is copied
    // once; without room for the copy, and for unaligned value vectors, the CUDA-core kernel takes the call.
    const int64_t ld = ((int64_t)N + 7) & ~7LL;
    const size_t copy_bytes = rhs_ok ? 0 : (((size_t)K * batch * ld * 2 + 255) & ~(size_t)255);
    bool simt = K == 0 || choice == 2 || !values_ok || ld > 0x7fffffff || (!rhs_ok && (ex.query || ex.caller_workspace)) ||
                copy_bytes > ((size_t)2 << 30);
    if (!simt) {
        if (choice == 1) {                                     // TMA row-gather producers
            if (ex.query) return 0;
            e = launch_sspmm_gather(a);
            return e == cudaSuccess ? 0 : fail(e, "SpMM launch");
        }
        if (!rhs_ok) {
            a.N = (int)ld;
            a.rhs_stride = batch > 1 ? (int64_t)K * ld : 0;
        }
        // A copied operand stays with the row-gather kernel: like the CUDA-core kernel
        // it sums fp32 results in round-to-nearest (2048 x 4608 half full, N = 1001, distance from 64 bits: 1.3e-7, the matrix
        // unit's truncated sums over all of K 2.7e-6, the CUDA cores 8.5e-7; 172, 53 and 1863 us) and multiplies no
        // infinity of B by a zero that is not in the list.
        const bool block_ok = block_fits(a, rhs_ok);
        if (choice == 3 && !block_ok && rhs_ok) {
            set_error("block kernel needs 16-byte aligned output, a shared value array for batches and <= 2 GiB of scratch");
            return (int)cudaErrorInvalidValue;
        }
        long long nvec = ex.nvec;
        if (nvec < 0 && !ex.query && (choice == 0 || choice == 4)) nvec = lookup_nvec(row_offsets, m_vec, st);
        if (!rhs_ok && choice == 0 && sspmm_rows_reads_unaligned(a, nvec)) {
            a.N = N;                                           // rows of B where they lie
            e = launch_sspmm_rows_unaligned(a, nvec);
            return e == cudaSuccess ? 0 : fail(e, "SpMM launch");
        }
        const bool use_block = block_ok && (choice == 3 || (choice == 0 && nvec >= 0 && block_kernel_is_faster(nvec, a)));
        const size_t want = use_block ? sspmm_block_scratch_bytes(a) : sspmm_rows_scratch_bytes(a, nvec);
        if (ex.query) { *ex.query = want; return 0; }
        void* scratch = nullptr;
        size_t room = want;
        if (ex.caller_workspace) {
            room = ex.workspace_bytes;
            if (use_block) {
                const size_t need = (size_t)K * m_vec * V * sizeof(__half);
                if (room < need || !ex.workspace) {
                    set_error("workspace of %zu bytes is too small: the block kernel needs at least %zu (sspmm_workspace_bytes reports %zu)",
                              room, need, want);
                    return (int)cudaErrorInvalidValue;
                }
                scratch = ex.workspace;
            } else if (want && room >= want) {
                scratch = ex.workspace;                         // null or too small: long rows are not cut (slower)
            }
        } else if (copy_bytes + want) {
            keep_pool_memory();
            e = cudaMallocAsync(&scratch, copy_bytes + want, st);
            if (e != cudaSuccess) {
                if (rhs_ok) return fail(e, "scratch allocation for the SpMM");
                cudaGetLastError();
                simt = true;                                    // no room for the copy
                a.N = N; a.rhs_stride = rhs_stride;
            }
        }
        if (!simt) {
            e = cudaSuccess;
            uint8_t* rest = static_cast<uint8_t*>(scratch);
            if (copy_bytes) {
                SpmmArgs src = a;
                src.N = N; src.rhs_stride = rhs_stride;
                e = launch_align_rows(src, (int)ld, static_cast<__half*>(scratch));
                a.rhs = static_cast<const __half*>(scratch);
                rest += copy_bytes;
            }
            if (e == cudaSuccess) e = use_block ? launch_sspmm_block(a, rest, room) : launch_sspmm_rows(a, nvec, want ? rest : nullptr, true);
            if (scratch && !ex.caller_workspace) cudaFreeAsync(scratch, st);
            return e == cudaSuccess ? 0 : fail(e, "SpMM launch");
        }
    }
    if (ex.query) return 0;
    e = launch_sspmm_simt(a);
    return e == cudaSuccess ? 0 : fail(e, "SpMM launch");
}

// Host memory that kernels write the numbers to which the host waits for (counts of a compression): the copy that came after the
// scans, into pageable memory, took as long as they did.  64 slots, 256 KB, allocated at the first use; a compression
// holds one while it waits, and copies to its own memory when there is none.
class HostSlots {
public:
    static constexpr size_t kBytes = 4096;
    void* take() {
        std::lock_guard<std::mutex> lk(mu_);
        if (!base_ && !failed_) {
            void* p = nullptr;
            if (cudaHostAlloc(&p, 64 * kBytes, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) base_ = static_cast<uint8_t*>(p);
            else { cudaGetLastError(); failed_ = true; }
        }
        if (!base_ || used_ == ~0ull) return nullptr;
        int k = 0;
        while (used_ >> k & 1ull) ++k;
        used_ |= 1ull << k;
        return base_ + k * kBytes;
    }
    void give_back(void* slot) {
        if (!slot) return;
        std::lock_guard<std::mutex> lk(mu_);
        used_ &= ~(1ull << ((static_cast<uint8_t*>(slot) - base_) / kBytes));
    }
private:
    std::mutex mu_;
    uint8_t* base_ = nullptr;
    unsigned long long used_ = 0;
    bool failed_ = false;
};
static HostSlots g_slots;
struct HostSlot {
    void* const at = g_slots.take();
    ~HostSlot() { g_slots.give_back(at); }
    HostSlot() = default;
    HostSlot(const HostSlot&) = delete;
    HostSlot& operator=(const HostSlot&) = delete;
};

}  // namespace sspmm_b200

using namespace sspmm_b200;

struct svc_job {
    SvcProblem p;
    SvcScratch s;
    bool with_values;
    long long nvec;
    long long table_ints;
    long long class_groups[kSvcSegs];      // groups per list segment; [0] = groups whose ascending order is exact
    int device;
    cudaStream_t stream;
};

struct svc_batch_job {
    int count, V;
    long long rows, entries, vec_rows;
    bool with_values;
    svc_job* inner;              // the compression of the stacked matrix
    void* block;                 // table, cuts and the stacked CSR
    SvcBatchEntry* d_tab;
    long long* d_cuts;
    cudaStream_t stream;
};

// The operands whose products with N columns work on a copy, and where it goes in room.
static int collect_copies(int count, const sspmm_dense_operand* operands, int N, void* room, SpmmArgs* a, __half** at, int* made, int64_t* offsets,
                          int64_t* bytes) {
    if (count < 0 || count > kMaxCopies || !operands || !offsets || !bytes) { set_error("null pointer or more than %d operands", kMaxCopies); return (int)cudaErrorInvalidValue; }
    const int choice = g_kernel_choice.load();
    int64_t room_for = 0;
    int copies = 0;
    for (int k = 0; k < count; ++k) {
        const sspmm_dense_operand& o = operands[k];
        offsets[k] = -1;
        if ((o.vec_length != 8 && o.vec_length != 16) || o.pieces < 1 || o.pieces > kMaxPieces || o.m_vec <= 0 || o.K <= 0 || N <= 0 || N % 8 != 0 ||
            o.m_vec > 0x7fffffff / o.vec_length / o.pieces || !o.row_offsets || !o.nvec || !o.column_indices || !o.values_f16 ||
            !aligned16(o.values_f16) || choice == 1 || choice == 2 || choice == 4)
            continue;
        SpmmArgs& s = a[copies];
        s = SpmmArgs{};
        s.m_vec = o.m_vec; s.V = o.vec_length; s.N = N; s.n_out = N; s.K = o.K;
        s.row_indices = nullptr; s.row_offsets = o.row_offsets[0]; s.column_indices = o.column_indices;
        s.values = static_cast<const __half*>(o.values_f16); s.rhs = s.values;
        s.out = room; s.out_f16 = true; s.bias = nullptr; s.batch = 1;
        s.values_stride = 0; s.rhs_stride = 0; s.out_stride = 0; s.stream = nullptr;
        // every piece would go to the block kernel by itself
        bool block = true;
        int64_t total = 0;
        for (int i = 0; i < o.pieces && block; ++i) {
            block = o.row_offsets[i] && o.nvec[i] >= 0 && total + o.nvec[i] <= 0x7fffffffLL && sspmm_block_scratch_bytes(s) <= ((size_t)2 << 30) &&
                    (choice == 3 || block_kernel_is_faster(o.nvec[i], s));
            s.piece_offsets[i] = o.row_offsets[i];
            s.piece_first[i] = (int)total;
            total += o.nvec[i];
        }
        if (!block) continue;
        s.m_vec = o.pieces * o.m_vec;
        s.pieces = o.pieces;
        if (sspmm_block_scratch_bytes(s) > ((size_t)2 << 30)) continue;
        offsets[k] = room_for;
        at[copies] = reinterpret_cast<__half*>(static_cast<uint8_t*>(room) + room_for);
        room_for += (int64_t)(((size_t)o.K * s.m_vec * s.V * sizeof(__half) + 255) & ~(size_t)255);
        ++copies;
    }
    *bytes = room_for;
    *made = copies;
    if (room && reinterpret_cast<uintptr_t>(room) % 256 != 0) { set_error("copies need room on a 256-byte boundary"); return (int)cudaErrorInvalidValue; }
    return 0;
}

// First half of a compression: counting and scans are enqueued.  slot: host memory for the totals, or null.
static int svc_count(int M, int K, int vec_length, const int* d_csr_row_ptr, const int* d_csr_col_idx, const void* d_csr_values_f16, void* stream,
                     void* slot, svc_job** job) {
    if (vec_length != 8 && vec_length != 16) {
        set_error("vec_length must be 8 or 16 (got %d)", vec_length);
        return (int)cudaErrorInvalidValue;
    }
    if (M < 0 || K < 0) { set_error("negative dimension"); return (int)cudaErrorInvalidValue; }
    if (K > kSvcMaxK) {
        set_error("K = %d exceeds the supported maximum of %d columns", K, kSvcMaxK);
        return (int)cudaErrorInvalidValue;
    }
    // d_csr_col_idx may be NULL when the matrix has no entries (it is then never read)
    if (!d_csr_row_ptr) { set_error("null CSR row pointer"); return (int)cudaErrorInvalidValue; }
    svc_job* j = new (std::nothrow) svc_job();
    if (!j) return (int)cudaErrorMemoryAllocation;
    memset(j, 0, sizeof *j);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    j->stream = st;
    cudaGetDevice(&j->device);
    j->p.M = M; j->p.K = K; j->p.V = vec_length; j->p.m_vec = (M + vec_length - 1) / vec_length;
    j->p.row_ptr = d_csr_row_ptr; j->p.col_idx = d_csr_col_idx;
    j->p.vals = static_cast<const __half*>(d_csr_values_f16);
    j->with_values = d_csr_values_f16 != nullptr;
    const size_t mv = (size_t)j->p.m_vec;
    // one allocation: vec_ptr[mv+1] | mode[mv] | tbl_len[mv] | class_list[mv] | queue[8] | pad | tbl_off[mv+1] | totals
    const size_t ints = (mv + 1) + mv + mv + mv + 8;
    const size_t ints_padded = (ints + 3) & ~(size_t)3;
    const size_t scan_blocks = (size_t)svc_scan_blocks((long long)mv);
    const size_t bytes = ints_padded * 4 + (mv + 1 + kSvcTotals + scan_blocks * kSvcScanFields) * 8;
    void* base = nullptr;
    keep_pool_memory();
    cudaError_t e = cudaMallocAsync(&base, bytes, st);
    if (e != cudaSuccess) { delete j; return fail(e, "scratch allocation"); }
    j->s.vec_ptr = static_cast<int*>(base);
    j->s.mode = j->s.vec_ptr + mv + 1;
    j->s.tbl_len = j->s.mode + mv;
    j->s.class_list = j->s.tbl_len + mv;
    j->s.queue = j->s.class_list + mv;
    j->s.tbl_off = reinterpret_cast<long long*>(static_cast<int*>(base) + ints_padded);
    j->s.totals = j->s.tbl_off + mv + 1;
    j->s.block_sums = j->s.totals + kSvcTotals;
    j->s.tables = nullptr;
    j->s.host_totals = static_cast<long long*>(slot);
    e = svc_count_and_scan(j->p, j->s, j->with_values, st);
    if (e != cudaSuccess) {
        if (slot) cudaStreamSynchronize(st);          // what was launched may write to the slot
        cudaFreeAsync(base, st);
        delete j;
        return fail(e, "SVC counting pass");
    }
    *job = j;
    return 0;
}

// Second half: waits for the totals, and checks them.  The job is gone when this fails.
static int svc_counted(svc_job* j, const void* slot, cudaStream_t st) {
    long long totals[kSvcTotals] = {0};
    cudaError_t e = slot ? cudaSuccess : cudaMemcpyAsync(totals, j->s.totals, sizeof totals, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && slot) memcpy(totals, slot, sizeof totals);
    j->s.host_totals = nullptr;
    const int bad = (int)totals[2 + kSvcSegs];
    if (e != cudaSuccess || bad || totals[0] > 0x7fffffffLL) {
        cudaFreeAsync(j->s.vec_ptr, st);
        delete j;
        if (e != cudaSuccess) return fail(e, "SVC counting pass");
        if (bad) set_error("CSR column id outside [0, K)");
        else set_error("more than 2^31-1 vectors");
        return (int)cudaErrorInvalidValue;
    }
    j->nvec = totals[0];
    j->table_ints = totals[1];
    for (int c = 0; c < kSvcSegs; ++c) j->class_groups[c] = totals[2 + c];
    return 0;
}

extern "C" {

int sspmm_f16_f32(int m_vec, int vec_length, int N, int K, const int* row_indices, const int* row_offsets,
                  const int* column_indices, const void* values_f16, const void* rhs_f16, float* out_f32,
                  void* stream) {
    return spmm_entry(m_vec, vec_length, N, K, 1, row_indices, row_offsets, column_indices, values_f16, 0, rhs_f16, 0,
                      out_f32, 0, false, stream);
}

int sspmm_f16_f16(int m_vec, int vec_length, int N, int K, const int* row_indices, const int* row_offsets,
                  const int* column_indices, const void* values_f16, const void* rhs_f16, void* out_f16, void* stream) {
    return spmm_entry(m_vec, vec_length, N, K, 1, row_indices, row_offsets, column_indices, values_f16, 0, rhs_f16, 0,
                      out_f16, 0, true, stream);
}

int sspmm_f16_f16_batched(int m_vec, int vec_length, int N, int K, int batch, const int* row_indices,
                          const int* row_offsets, const int* column_indices, const void* values_f16,
                          int64_t values_stride, const void* rhs_f16, int64_t rhs_stride, void* out_f16,
                          int64_t out_stride, void* stream) {
    return spmm_entry(m_vec, vec_length, N, K, batch, row_indices, row_offsets, column_indices, values_f16,
                      values_stride, rhs_f16, rhs_stride, out_f16, out_stride, true, stream);
}

int sspmm_counted(int m_vec, int vec_length, int N, int K, int batch, int64_t nvec, const int* row_indices, const int* row_offsets,
                  const int* column_indices, const void* values_f16, int64_t values_stride, const void* rhs_f16, int64_t rhs_stride,
                  const void* bias_f16, void* out, int64_t out_stride, int out_is_f16, void* stream) {
    if (nvec < 0) { g_err[0] = 0; set_error("nvec must be >= 0"); return (int)cudaErrorInvalidValue; }
    SpmmExtra ex;
    ex.nvec = nvec; ex.bias = bias_f16;
    return spmm_entry(m_vec, vec_length, N, K, batch, row_indices, row_offsets, column_indices, values_f16, values_stride, rhs_f16,
                      rhs_stride, out, out_stride, out_is_f16 != 0, stream, ex);
}

int sspmm_counted_sum(int m_vec, int vec_length, int N, int K, int64_t nvec, const int* row_indices, const int* row_offsets,
                      const int* column_indices, const void* values_f16, const void* rhs_f16, const void* bias_f16, const void* add_f16,
                      void* out_f16, void* stream, int* taken) {
    g_err[0] = 0;
    if (!taken || nvec < 0) { set_error("null pointer or negative nvec"); return (int)cudaErrorInvalidValue; }
    *taken = 0;
    const int choice = g_kernel_choice.load();
    if ((vec_length != 8 && vec_length != 16) || m_vec <= 0 || N <= 0 || K <= 0 || m_vec > 0x7fffffff / vec_length || N % 8 != 0 || !row_offsets ||
        !column_indices || !values_f16 || !rhs_f16 || !add_f16 || !out_f16 || !aligned16(values_f16) || !aligned16(rhs_f16) || !aligned16(add_f16) ||
        !aligned16(out_f16) || choice == 1 || choice == 2)
        return 0;
    SpmmArgs a;
    a.m_vec = m_vec; a.V = vec_length; a.N = N; a.n_out = N; a.K = K;
    a.row_indices = row_indices; a.row_offsets = row_offsets; a.column_indices = column_indices;
    a.values = static_cast<const __half*>(values_f16); a.rhs = static_cast<const __half*>(rhs_f16);
    a.out = out_f16; a.out_f16 = true; a.bias = static_cast<const __half*>(bias_f16); a.add = static_cast<const __half*>(add_f16); a.batch = 1;
    a.values_stride = 0; a.rhs_stride = 0; a.out_stride = 0;
    a.stream = static_cast<cudaStream_t>(stream);
    // the kernel that sspmm_counted takes
    const bool fits = block_fits(a, true);
    cudaError_t e;
    if (fits && (choice == 3 || (choice == 0 && block_kernel_is_faster(nvec, a)))) {
        void* scratch = nullptr;
        const size_t bytes = sspmm_block_scratch_bytes(a);
        keep_pool_memory();
        e = cudaMallocAsync(&scratch, bytes, a.stream);
        if (e != cudaSuccess) { cudaGetLastError(); return 0; }
        e = launch_sspmm_block(a, scratch, bytes);
        cudaFreeAsync(scratch, a.stream);
    } else {
        if (choice == 3 || sspmm_rows_may_be_long(a, nvec)) return 0;
        e = launch_sspmm_rows_set(&a, 1, nvec);
    }
    if (e != cudaSuccess) return fail(e, "SpMM launch");
    *taken = 1;
    return 0;
}

int sspmm_dense_copies(int count, const sspmm_dense_operand* operands, int N, void* room, int64_t* offsets, int64_t* bytes, void* stream) {
    g_err[0] = 0;
    SpmmArgs a[kMaxCopies];
    __half* at[kMaxCopies];
    int copies = 0;
    const int rc = collect_copies(count, operands, N, room, a, at, &copies, offsets, bytes);
    if (rc != 0 || !room || copies == 0) return rc;
    const cudaError_t e = launch_expand_set(a, at, copies, static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? 0 : fail(e, "dense copies");
}

int sspmm_of_copy(int m_vec, int vec_length, int N, int K, const void* copy_f16, const void* rhs_f16, const void* bias_f16, const void* add_f16,
                  void* out_f16, void* stream) {
    g_err[0] = 0;
    if ((vec_length != 8 && vec_length != 16) || m_vec <= 0 || N <= 0 || K <= 0 || m_vec > 0x7fffffff / vec_length || N % 8 != 0 || !copy_f16 || !rhs_f16 ||
        !out_f16 || !aligned16(copy_f16) || !aligned16(rhs_f16) || !aligned16(add_f16) || !aligned16(out_f16)) {
        set_error("a product of a dense copy needs N %% 8 == 0 and 16-byte aligned operands");
        return (int)cudaErrorInvalidValue;
    }
    SpmmArgs a;
    a.m_vec = m_vec; a.V = vec_length; a.N = N; a.n_out = N; a.K = K;
    a.row_indices = nullptr; a.row_offsets = nullptr; a.column_indices = nullptr; a.values = nullptr;
    a.rhs = static_cast<const __half*>(rhs_f16);
    a.out = out_f16; a.out_f16 = true; a.bias = static_cast<const __half*>(bias_f16); a.add = static_cast<const __half*>(add_f16); a.batch = 1;
    a.values_stride = 0; a.rhs_stride = 0; a.out_stride = 0;
    a.stream = static_cast<cudaStream_t>(stream);
    a.copy = static_cast<const __half*>(copy_f16);
    const size_t bytes = sspmm_block_scratch_bytes(a);              // partial tiles of a cut K range
    void* scratch = nullptr;
    cudaError_t e = cudaSuccess;
    if (bytes) {
        keep_pool_memory();
        e = cudaMallocAsync(&scratch, bytes, a.stream);
        if (e != cudaSuccess) return fail(e, "scratch allocation for the SpMM");
    }
    e = launch_sspmm_block(a, scratch, bytes);
    if (scratch) cudaFreeAsync(scratch, a.stream);
    return e == cudaSuccess ? 0 : fail(e, "SpMM launch");
}

int sspmm_stacked(int pieces, int m_vec, int vec_length, int N, int K, const int64_t* nvec, const int* const* row_indices,
                  const int* const* row_offsets, const int* column_indices, const void* values_f16, const void* rhs_f16,
                  const void* bias_f16, void* out, int out_is_f16, void* stream, int* taken) {
    g_err[0] = 0;
    if (!taken || !nvec || !row_offsets || pieces < 1) { set_error("null pointer or no pieces"); return (int)cudaErrorInvalidValue; }
    *taken = 0;
    const int choice = g_kernel_choice.load();
    const int V = vec_length;
    if (pieces > kMaxPieces || (V != 8 && V != 16) || m_vec <= 0 || N <= 0 || K <= 0 || m_vec > 0x7fffffff / V / pieces || N % 8 != 0 ||
        !column_indices || !values_f16 || !rhs_f16 || !out || !aligned16(values_f16) || !aligned16(rhs_f16) || !aligned16(out) ||
        choice == 1 || choice == 2)
        return 0;
    SpmmArgs a;
    a.m_vec = pieces * m_vec; a.V = V; a.N = N; a.n_out = N; a.K = K;
    a.row_indices = nullptr; a.row_offsets = row_offsets[0]; a.column_indices = column_indices;
    a.values = static_cast<const __half*>(values_f16); a.rhs = static_cast<const __half*>(rhs_f16);
    a.out = out; a.out_f16 = out_is_f16 != 0; a.bias = static_cast<const __half*>(bias_f16); a.batch = 1;
    a.values_stride = 0; a.rhs_stride = 0; a.out_stride = 0;
    a.stream = static_cast<cudaStream_t>(stream);
    a.pieces = pieces;
    SpmmArgs each[kMaxPieces];
    int64_t total = 0;
    // The pieces go to the kernel that they would go to one by one, not to the one that is faster for all of them: the block kernel
    // multiplies an infinity of rhs by zeros that are in no list, and a call's results must not depend on being stacked.
    int block = 0;
    for (int i = 0; i < pieces; ++i) {
        if (!row_offsets[i] || nvec[i] < 0 || total + nvec[i] > 0x7fffffffLL) return 0;
        a.piece_offsets[i] = row_offsets[i];
        a.piece_first[i] = (int)total;
        SpmmArgs& s = each[i];
        s = a;
        s.pieces = 1; s.m_vec = m_vec;
        s.row_indices = row_indices ? row_indices[i] : nullptr; s.row_offsets = row_offsets[i];
        s.column_indices = column_indices + total; s.values = a.values + total * V;
        s.out = static_cast<uint8_t*>(out) + (size_t)i * m_vec * V * N * (out_is_f16 ? 2 : 4);
        s.bias = a.bias ? a.bias + (size_t)i * m_vec * V : nullptr;
        if (block_fits(s, true) && (choice == 3 || (choice == 0 && block_kernel_is_faster(nvec[i], s)))) ++block;
        else if (choice == 3 || sspmm_rows_may_be_long(s, nvec[i])) return 0;    // not in a launch of several products
        total += nvec[i];
    }
    if (block != 0 && (block != pieces || !block_fits(a, true))) return 0;
    cudaError_t e;
    if (block) {
        void* scratch = nullptr;
        const size_t bytes = sspmm_block_scratch_bytes(a);
        keep_pool_memory();
        e = cudaMallocAsync(&scratch, bytes, a.stream);
        if (e != cudaSuccess) { cudaGetLastError(); return 0; }
        e = launch_sspmm_block(a, scratch, bytes);
        cudaFreeAsync(scratch, a.stream);
    } else {
        e = launch_sspmm_rows_set(each, pieces, total);
    }
    if (e != cudaSuccess) return fail(e, "SpMM launch");
    *taken = 1;
    return 0;
}

int sspmm_workspace_bytes(int m_vec, int vec_length, int N, int K, int64_t nvec, int out_is_f16, int64_t* bytes) {
    if (!bytes || nvec < 0) { g_err[0] = 0; set_error("bytes must be non-null and nvec >= 0"); return (int)cudaErrorInvalidValue; }
    SpmmExtra ex;
    size_t q = 0;
    ex.nvec = nvec; ex.query = &q;
    // aligned dummy operands: only sizes and alignment enter the choice of kernel
    void* dummy = reinterpret_cast<void*>(uintptr_t(256));
    const int rc = spmm_entry(m_vec, vec_length, N, K, 1, nullptr, nullptr, nullptr, dummy, 0, dummy, 0, dummy, 0, out_is_f16 != 0,
                              nullptr, ex);
    *bytes = (int64_t)q;
    return rc;
}

int sspmm_f16_f16_ws(int m_vec, int vec_length, int N, int K, const int* row_indices, const int* row_offsets,
                     const int* column_indices, const void* values_f16, const void* rhs_f16, void* out_f16, int64_t nvec,
                     void* workspace, int64_t workspace_bytes, void* stream) {
    if (nvec < 0 || workspace_bytes < 0) { g_err[0] = 0; set_error("nvec and workspace_bytes must be >= 0"); return (int)cudaErrorInvalidValue; }
    SpmmExtra ex;
    ex.nvec = nvec; ex.workspace = workspace; ex.workspace_bytes = (size_t)workspace_bytes; ex.caller_workspace = true;
    return spmm_entry(m_vec, vec_length, N, K, 1, row_indices, row_offsets, column_indices, values_f16, 0, rhs_f16, 0, out_f16, 0,
                      true, stream, ex);
}

int sspmm_set_kernel(int which) {
    if (which < 0 || which > 5) {
        set_error("kernel selector must be 0..5");
        return (int)cudaErrorInvalidValue;
    }
    sspmm_block_allow_pairs(which != 5);
    g_kernel_choice.store(which == 5 ? 3 : which);
    return 0;
}

int sspmm_device_status(int* status) {
    g_err[0] = 0;
    if (!status) return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return fail(e, "device synchronize");
    e = cudaMemcpyFromSymbol(status, g_device_status, sizeof(int));
    if (e != cudaSuccess) return fail(e, "status read");
    if (*status != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int));
        if (e != cudaSuccess) return fail(e, "status clear");
    }
    return 0;
}

int sspmm_selftest_wait_expiry(long long limit_cycles, int* gave_up) {
    g_err[0] = 0;
    if (!gave_up || limit_cycles <= 0 || limit_cycles > kDefaultWaitCycleLimit) {
        set_error("limit_cycles must be in (0, %lld] and gave_up non-null", kDefaultWaitCycleLimit);
        return (int)cudaErrorInvalidValue;
    }
    *gave_up = -1;
    int* d_flag = nullptr;
    cudaError_t e = cudaDeviceSynchronize();                       // no other kernel of ours sees the short limit
    if (e == cudaSuccess) e = cudaMalloc(&d_flag, sizeof(int));
    if (e != cudaSuccess) return fail(e, "self test set-up");
    e = cudaMemcpyToSymbol(g_wait_cycle_limit, &limit_cycles, sizeof(long long));
    if (e == cudaSuccess) {
        wait_expiry_selftest_kernel<<<1, 32>>>(d_flag);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        const long long back = kDefaultWaitCycleLimit;
        const cudaError_t e2 = cudaMemcpyToSymbol(g_wait_cycle_limit, &back, sizeof(long long));
        if (e == cudaSuccess) e = e2;
    }
    if (e == cudaSuccess) e = cudaMemcpy(gave_up, d_flag, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d_flag);
    return e == cudaSuccess ? 0 : fail(e, "wait-expiry self test");
}

int svc_begin(int M, int K, int vec_length, const int* d_csr_row_ptr, const int* d_csr_col_idx,
              const void* d_csr_values_f16, void* stream, svc_job** job, int64_t* nvec) {
    g_err[0] = 0;
    if (!job || !nvec) { set_error("null output pointer"); return (int)cudaErrorInvalidValue; }
    *job = nullptr;
    const HostSlot slot;
    svc_job* j = nullptr;
    int rc = svc_count(M, K, vec_length, d_csr_row_ptr, d_csr_col_idx, d_csr_values_f16, stream, slot.at, &j);
    if (rc == 0) rc = svc_counted(j, slot.at, static_cast<cudaStream_t>(stream));
    if (rc != 0) return rc;
    *nvec = j->nvec;
    *job = j;
    return 0;
}

int svc_finish(svc_job* j, int* d_vec_row_ptr, int* d_vec_col, void* d_vec_values_f16, void* stream) {
    g_err[0] = 0;
    if (!j || !d_vec_row_ptr || (j->nvec > 0 && !d_vec_col)) { set_error("null pointer"); return (int)cudaErrorInvalidValue; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaSuccess;
    if (j->nvec == 0) {
        e = cudaMemcpyAsync(d_vec_row_ptr, j->s.vec_ptr, ((size_t)j->p.m_vec + 1) * 4, cudaMemcpyDeviceToDevice, st);
        return e == cudaSuccess ? 0 : fail(e, "row pointer copy");
    }
    __half* ov = j->with_values ? static_cast<__half*>(d_vec_values_f16) : nullptr;
    j->p.zero_values = aligned16(ov);
    if (ov && !j->p.zero_values) {
        e = cudaMemsetAsync(ov, 0, (size_t)j->nvec * j->p.V * sizeof(__half), st);
        if (e != cudaSuccess) return fail(e, "value clear");
    }
    if (j->table_ints > 0 && !j->s.tables) {
        e = cudaMallocAsync(reinterpret_cast<void**>(&j->s.tables), (size_t)j->table_ints * 4, st);
        if (e != cudaSuccess) return fail(e, "table scratch allocation");
    }
    e = svc_emit(j->p, j->s, j->class_groups, d_vec_row_ptr, d_vec_col, ov, st);
    if (e != cudaSuccess) return fail(e, "SVC emit");
    j->stream = st;
    return 0;
}

int svc_free(svc_job* j) {
    if (!j) return 0;
    if (j->s.tables) cudaFreeAsync(j->s.tables, j->stream);
    if (j->s.vec_ptr) cudaFreeAsync(j->s.vec_ptr, j->stream);
    delete j;
    return 0;
}

int svc_batch_begin(int count, int vec_length, const int* M, const int* K, const int* nnz,
                    const int* const* d_csr_row_ptr, const int* const* d_csr_col_idx, const void* const* d_csr_values_f16,
                    void* stream, svc_batch_job** job, int64_t* nvec) {
    g_err[0] = 0;
    if (!job || !nvec) { set_error("null output pointer"); return (int)cudaErrorInvalidValue; }
    *job = nullptr;
    if (count <= 0 || !M || !K || !nnz || !d_csr_row_ptr || !d_csr_col_idx) {
        set_error("a batch needs at least one matrix and its size arrays");
        return (int)cudaErrorInvalidValue;
    }
    if (vec_length != 8 && vec_length != 16) {
        set_error("vec_length must be 8 or 16 (got %d)", vec_length);
        return (int)cudaErrorInvalidValue;
    }
    const int V = vec_length;
    std::vector<SvcBatchEntry> tab((size_t)count + 1);
    long long rows = 0, entries = 0, vec_rows = 0;
    int k_max = 0;
    bool with_values = d_csr_values_f16 != nullptr;
    for (int i = 0; i < count; ++i) {
        if (M[i] < 0 || K[i] < 0 || nnz[i] < 0 || !d_csr_row_ptr[i] || (nnz[i] > 0 && !d_csr_col_idx[i])) {
            set_error("matrix %d: bad size or null array", i);
            return (int)cudaErrorInvalidValue;
        }
        if (with_values && nnz[i] > 0 && !d_csr_values_f16[i]) with_values = false;
        const long long mv = (M[i] + V - 1) / V;
        tab[i] = SvcBatchEntry{d_csr_row_ptr[i], d_csr_col_idx[i], with_values ? static_cast<const __half*>(d_csr_values_f16[i]) : nullptr,
                               rows, entries, vec_rows, M[i], nnz[i]};
        rows += mv * V; entries += nnz[i]; vec_rows += mv;
        if (K[i] > k_max) k_max = K[i];
    }
    tab[count] = SvcBatchEntry{nullptr, nullptr, nullptr, rows, entries, vec_rows, 0, 0};
    if (rows >= 0x7fffffffLL || entries >= 0x7fffffffLL) {
        set_error("stacked batch does not fit 32-bit indices (%lld rows, %lld entries)", rows, entries);
        return (int)cudaErrorInvalidValue;
    }
    if (k_max > kSvcMaxK) {
        set_error("K = %d exceeds the supported maximum of %d columns", k_max, kSvcMaxK);
        return (int)cudaErrorInvalidValue;
    }
    svc_batch_job* b = new (std::nothrow) svc_batch_job();
    if (!b) return (int)cudaErrorMemoryAllocation;
    b->count = count; b->V = V; b->rows = rows; b->entries = entries; b->vec_rows = vec_rows; b->with_values = with_values;
    b->inner = nullptr; b->block = nullptr;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // one allocation: table | cuts[count+1] (int64) | stacked row_ptr | stacked col | stacked values
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t off_cuts = up(tab.size() * sizeof(SvcBatchEntry));
    const size_t off_ptr = off_cuts + up(((size_t)count + 1) * 8);
    const size_t off_col = off_ptr + up(((size_t)rows + 1) * 4);
    const size_t off_val = off_col + up((size_t)entries * 4);
    const size_t total = off_val + (with_values ? up((size_t)entries * 2) : 0);
    keep_pool_memory();
    cudaError_t e = cudaMallocAsync(&b->block, total, st);
    if (e != cudaSuccess) { delete b; return fail(e, "batch scratch allocation"); }
    uint8_t* base = static_cast<uint8_t*>(b->block);
    b->d_tab = reinterpret_cast<SvcBatchEntry*>(base);
    b->d_cuts = reinterpret_cast<long long*>(base + off_cuts);
    int* s_ptr = reinterpret_cast<int*>(base + off_ptr);
    int* s_col = reinterpret_cast<int*>(base + off_col);
    __half* s_val = with_values ? reinterpret_cast<__half*>(base + off_val) : nullptr;
    e = svc_stack(tab.data(), b->d_tab, count, rows, entries, s_ptr, s_col, s_val, st);
    // the cuts go to the slot behind the totals, where there is room, and one wait is for both
    const HostSlot slot;
    constexpr size_t kCutsAt = 256;
    static_assert(kSvcTotals * 8 <= kCutsAt, "cuts behind the totals");
    long long* const near = slot.at && kCutsAt + ((size_t)count + 1) * 8 <= HostSlots::kBytes
                                ? reinterpret_cast<long long*>(static_cast<uint8_t*>(slot.at) + kCutsAt) : nullptr;
    int rc = 0;
    if (e == cudaSuccess) {
        rc = svc_count((int)rows, k_max, V, s_ptr, s_col, s_val, stream, slot.at, &b->inner);
        if (rc == 0) {
            e = svc_batch_cuts(b->d_tab, count, b->inner->s.vec_ptr, b->d_cuts, near, st);
            rc = svc_counted(b->inner, slot.at, st);
            if (rc != 0) b->inner = nullptr;
        }
        std::vector<long long> copied;
        const long long* cuts = near;
        if (e == cudaSuccess && rc == 0 && !near) {
            copied.resize((size_t)count + 1);
            e = cudaMemcpyAsync(copied.data(), b->d_cuts, copied.size() * 8, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            cuts = copied.data();
        }
        if (e == cudaSuccess && rc == 0)
            for (int i = 0; i < count; ++i) nvec[i] = cuts[i + 1] - cuts[i];
    }
    if (e != cudaSuccess || rc != 0) {
        if (b->inner) svc_free(b->inner);
        cudaFreeAsync(b->block, st);
        delete b;
        return rc != 0 ? rc : fail(e, "batch stacking");
    }
    b->stream = st;
    *job = b;
    return 0;
}

int svc_batch_finish(svc_batch_job* b, int* d_vec_row_ptr, int* d_vec_col, void* d_vec_values_f16, void* stream) {
    g_err[0] = 0;
    if (!b || !d_vec_row_ptr) { set_error("null pointer"); return (int)cudaErrorInvalidValue; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    svc_job* j = b->inner;
    // vector row pointers of each matrix, rebased to start at 0, one after another
    cudaError_t e = svc_batch_row_ptrs(b->d_tab, b->count, b->vec_rows, j->s.vec_ptr, b->d_cuts, d_vec_row_ptr, st);
    if (e != cudaSuccess) return fail(e, "row pointer rebase");
    if (j->nvec == 0) return 0;
    if (!d_vec_col) { set_error("null pointer"); return (int)cudaErrorInvalidValue; }
    __half* ov = j->with_values ? static_cast<__half*>(d_vec_values_f16) : nullptr;
    j->p.zero_values = aligned16(ov);
    if (ov && !j->p.zero_values) {
        e = cudaMemsetAsync(ov, 0, (size_t)j->nvec * j->p.V * sizeof(__half), st);
        if (e != cudaSuccess) return fail(e, "value clear");
    }
    if (j->table_ints > 0 && !j->s.tables) {
        e = cudaMallocAsync(reinterpret_cast<void**>(&j->s.tables), (size_t)j->table_ints * 4, st);
        if (e != cudaSuccess) return fail(e, "table scratch allocation");
    }
    e = svc_emit(j->p, j->s, j->class_groups, nullptr, d_vec_col, ov, st);
    if (e != cudaSuccess) return fail(e, "SVC emit");
    j->stream = st;
    b->stream = st;
    return 0;
}

int svc_batch_replayed_rows(svc_batch_job* b, int64_t* rows) {
    if (!b || !b->inner) return (int)cudaErrorInvalidValue;
    return svc_replayed_rows(b->inner, rows);
}

int svc_batch_free(svc_batch_job* b) {
    if (!b) return 0;
    if (b->inner) svc_free(b->inner);
    if (b->block) cudaFreeAsync(b->block, b->stream);
    delete b;
    return 0;
}

int svc_replayed_rows(svc_job* j, int64_t* rows) {
    g_err[0] = 0;
    if (!j || !rows) return (int)cudaErrorInvalidValue;
    *rows = 0;
    for (int c = 1; c < kSvcSegs; ++c) *rows += j->class_groups[c];       // every class but "ascending"
    return 0;
}

int sspmm_sorted_row_swizzle(int m_vec, const int* d_row_offsets, int* d_row_indices, void* stream) {
    g_err[0] = 0;
    if (m_vec < 0 || (m_vec > 0 && (!d_row_offsets || !d_row_indices))) {
        set_error("bad argument");
        return (int)cudaErrorInvalidValue;
    }
    if (m_vec == 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (m_vec <= kSwizzleRankLimit) {
        row_swizzle_kernel<<<(m_vec + 255) / 256, 256, 0, st>>>(m_vec, d_row_offsets, d_row_indices);
        cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? 0 : fail(e, "row swizzle launch");
    }
    long long padded = 1;
    while (padded < m_vec) padded <<= 1;
    unsigned long long* keys = nullptr;
    keep_pool_memory();
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&keys), (size_t)padded * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return fail(e, "scratch allocation for the row order");
    const unsigned blocks = (unsigned)((padded + 255) / 256);
    swizzle_keys_kernel<<<blocks, 256, 0, st>>>(m_vec, padded, d_row_offsets, keys);
    for (long long k = 2; k <= padded; k <<= 1)
        for (long long j = k >> 1; j > 0; j >>= 1) swizzle_bitonic_kernel<<<blocks, 256, 0, st>>>(padded, j, k, keys);
    swizzle_write_kernel<<<(m_vec + 255) / 256, 256, 0, st>>>(m_vec, keys, d_row_indices);
    e = cudaGetLastError();
    cudaFreeAsync(keys, st);
    return e == cudaSuccess ? 0 : fail(e, "row swizzle launch");
}

const char* sspmm_last_error_string(void) { return g_err; }
const char* sspmm_version(void) { return "sspmm_b200 0.1 sm_100a"; }

}  // extern "C"
