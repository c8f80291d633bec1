// Internal launcher interface shared by the kernel translation units and the C ABI.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <atomic>

namespace sspmm_b200 {

constexpr int kMaxPieces = 4;

struct SpmmArgs {
    int m_vec;                 // vector rows
    int V;                     // rows per vector (8 or 16)
    int N;                     // columns of the dense operand as it is read (its row pitch)
    int n_out;                 // columns of the output (its row pitch); N unless the dense operand is an aligned copy
    int K;                     // rows of the dense operand
    const int* row_indices;    // optional scheduling order of vector rows (may be null)
    const int* row_offsets;    // [m_vec + 1]
    const int* column_indices; // [nvec]
    const __half* values;      // [nvec * V]
    const __half* rhs;         // [K * N] row-major
    void* out;                 // [m_vec * V * N] row-major, fp32 or fp16
    bool out_f16;
    const __half* bias;        // per row of the output, added before the conversion; may be null
    const __half* add = nullptr;   // like the output, added as well (fp16 results of one product; block kernel and launch_sspmm_rows_set)
    // batching (one launch, grid z-less: tiles enumerate the batch too)
    int batch;                 // >= 1
    int64_t values_stride;     // elements between batches (0 = shared)
    int64_t rhs_stride;
    int64_t out_stride;
    cudaStream_t stream;
    // The operand may be several of one height, one below the other, that share column_indices and values but keep their own row
    // pointers (block kernel only): piece p starts at vector piece_first[p].  pieces <= 1: row_offsets are those of the operand.
    int pieces = 1;
    const int* piece_offsets[kMaxPieces] = {};
    int piece_first[kMaxPieces] = {};
    // Block kernel: the dense transposed copy [K][m_vec*V] of the operand (launch_expand_set); null: it makes its own from the operand.
    const __half* copy = nullptr;
};

// tcgen05 row-gather kernel.  Requires N % 8 == 0, 16-byte aligned rhs/values.
cudaError_t launch_sspmm_gather(const SpmmArgs& a);
// Row-gather kernel: N % 8 == 0, rhs and values 16-byte aligned; any n_out <= N.
// scratch: null, or sspmm_rows_scratch_bytes() bytes when that is not 0 (long rows are then cut); nvec < 0: unknown.
size_t sspmm_rows_scratch_bytes(const SpmmArgs& a, long long nvec);
// spread: the warps are divided with a row in mind that is many times the mean, where there may be one.
cudaError_t launch_sspmm_rows(const SpmmArgs& a, long long nvec, void* scratch, bool spread);
// Whether there may be one.
bool sspmm_rows_may_be_long(const SpmmArgs& a, long long nvec);
// The same for an rhs on a 16-byte boundary whose N is not a multiple of 8, one product without a copy of rhs; whether a call is one for it.
bool sspmm_rows_reads_unaligned(const SpmmArgs& a, long long nvec);
cudaError_t launch_sspmm_rows_unaligned(const SpmmArgs& a, long long nvec);
// Several products with vectors of one length and outputs of one type in one launch; no scratch.  nvec: vectors of all of them.
constexpr int kRowsMaxSet = 8;
cudaError_t launch_sspmm_rows_set(const SpmmArgs* a, int count, long long nvec);
// How that launch divides the products: columns of a tile, warps that share an item (a vector row of a tile), items, CTAs.
struct RowsShape { int columns, warps; long long items, ctas; };
RowsShape sspmm_rows_set_shape(const SpmmArgs* a, int count, long long nvec);
// Copy of the dense operand with rows of `ld` columns (a multiple of 8, zeros in the columns added).
cudaError_t launch_align_rows(const SpmmArgs& a, int ld, __half* dst);
// tcgen05 block kernel on a dense transposed copy of A held in `scratch` (caller-owned, stream-ordered).
// sspmm_block_scratch_bytes(a) is what the kernel would like (copy of A + split-K partial tiles); with less
// (at least K * m_vec*V halfs) it runs without split-K.
size_t sspmm_block_scratch_bytes(const SpmmArgs& a);
cudaError_t launch_sspmm_block(const SpmmArgs& a, void* scratch, size_t scratch_bytes);
// Dense transposed copies of several operands (m_vec, V, K, column_indices, values and the row offsets of their pieces count) in one
// launch; at[i] holds K * m_vec*V halfs.
constexpr int kMaxCopies = 8;
cudaError_t launch_expand_set(const SpmmArgs* a, __half* const* at, int count, cudaStream_t stream);
// Allows (default) or forbids the CTA-pair variant of the block kernel.  Process-wide.
void sspmm_block_allow_pairs(bool allow);
// CUDA-core kernel without alignment requirements.
cudaError_t launch_sspmm_simt(const SpmmArgs& a);

// Per-device "already done" flags for one-time, per-device set-up (function
// attributes are per device).  Supports device ordinals 0..63.
class DeviceOnce {
public:
    bool done() const {
        int d = 0;
        cudaGetDevice(&d);
        return d >= 0 && d < 64 && (mask_.load(std::memory_order_acquire) >> d) & 1ull;
    }
    void mark() {
        int d = 0;
        cudaGetDevice(&d);
        if (d >= 0 && d < 64) mask_.fetch_or(1ull << d, std::memory_order_release);
    }
private:
    std::atomic<unsigned long long> mask_{0};
};

// Multiprocessor count of the current device (cached per device ordinal).
int current_device_sm_count();

// Records a message retrievable through sspmm_last_error_string().
void set_error(const char* fmt, ...);

}  // namespace sspmm_b200
