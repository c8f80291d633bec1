// Vector-sparse SpMM by rows, for operands whose dense tiles would be mostly padding and for products so small that
// start-up latency decides: every warp gathers the rows of B that a vector row names and multiplies them by itself.
//
// Same contract as the other SpMM kernels (reference entry: SSpMM/src/sspmm.cu:626-649).
//
// What bounds it: every vector moves a row of B from L2 to an SM for V output rows, so the work is 2 * nvec * N bytes
// of L2 reads, and a warp that waits for each of its reads in turn sees their full latency.  The split follows from
// that: sixteen independent warps per SM, each with two or three steps of sixteen gathered rows in flight.
// The arithmetic is 16 gathered rows per instruction (mma.m16n8k16, the transposed product
//   D[n][v] += B^T[n][k] * vals[k][v]);
// a tcgen05.mma of that depth holds its issuing thread for longer (about 130 cycles measured, plus 100 per commit) than
// this path needs for the whole 16-row step, and its accumulators would have to come back from tensor memory for every
// row.  A warp keeps its own ring of steps in shared memory, filled by cp.async (16 bytes per lane, eight lanes per 128
// bytes of a row of B) and read by ldmatrix, so that neither side has bank conflicts; loading the fragments straight
// into registers was tried and is bound by the L1 data stage (four rows of B per quarter warp fall on the same banks:
// 6.0 TB/s of gathers where the ring reaches 9 to 10).
//
// Measured (graph replays, against the former kernel that passed stages of 64 rows to tcgen05.mma): 512 x 512 at 70 %, N =
// 256: 5.4 us (12.7); 2048 x 512 at 90 %, V = 16, N = 256: 8.0 (16.6); 512 x 4608 at 90 %, N = 64: 7.5 (26.3), with clusters by
// what a full row would take (route) N = 56 4.7.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>

#include "launch.h"
#include "ptx.cuh"

namespace sspmm_b200 {
namespace rows {

constexpr int kWarps = 8;                 // per CTA
constexpr int kThreads = kWarps * 32;
constexpr int kStep = 16;                 // vectors per step
constexpr int kLightRow = 256;            // split launches: longest row that one warp does
constexpr int kMaxCluster = 8;
constexpr int kResident = 2;              // CTAs per SM: 16 warps with two or three steps in flight each

struct Problem {
    int m_vec, K, n_tiles;
    int N;                                // columns of C (and its row pitch)
    int ldb;                              // row pitch of B, a multiple of 8: columns [N, ldb) exist and are multiplied along
    long long items;                      // m_vec * n_tiles * batch
    const int* row_indices;
    const int* row_offsets;
    const int* col;
    const __half* values;
    const __half* rhs;
    const __half* bias;                   // per row of C, or null
    int64_t values_stride, rhs_stride, out_stride;
    int out_pieces;                       // rows of C start on 16-byte boundaries
    // split launches only (see sspmm_rows_split_kernel)
    int chunk;                            // vectors per part
    int cap_cut, cap_whole;               // room for parts of rows with several, and for rows that are one part
    int* header;                          // [0] parts of rows with several, [1] next row item, [2] rows that are one part
    int* arrivals;                        // [part][n_tile], at a row's part 0: its finished parts
    int4* entries;                        // vector row, first vector, vectors, parts of the row << 16 | number: cap_cut parts, cap_whole rows
    float* partial;                       // [part][n_tile][V][NT] sums, of rows with several parts only
};

// d += a * b of one instruction: 16 columns x 8 rows of C, 16 vectors deep.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, bool valid) {
    const uint32_t bytes = valid ? 16u : 0u;                       // 0: the destination is zero-filled, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_bytes(uint32_t dst, const void* src, uint32_t bytes) {      // up to 16 bytes, zeros after them
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t& r0, uint32_t& r1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}

struct Where { int row, j0, len, n0, batch; };      // row = -1: nothing to do

__device__ __forceinline__ Where locate(const Problem& p, long long T, int NT) {
    Where w;
    w.row = -1; w.j0 = 0; w.len = 0; w.n0 = 0; w.batch = 0;
    if (T >= p.items) return w;
    const int sched = (int)(T % p.m_vec);
    const int rest = (int)(T / p.m_vec);
    const int i = p.row_indices ? __ldg(p.row_indices + sched) : sched;
    if ((unsigned)i >= (unsigned)p.m_vec) return w;
    w.row = i;
    w.n0 = (rest % p.n_tiles) * NT;
    w.batch = rest / p.n_tiles;
    w.j0 = __ldg(p.row_offsets + i);
    w.len = max(0, __ldg(p.row_offsets + i + 1) - w.j0);
    return w;
}

// V rows per vector, H 64-column halves per tile.
// ROUND: every step is summed from zero and added to the accumulator by an fp32 addition that rounds to nearest (the
// instruction's own additions truncate, which adds up over a long row); fp32 results only, fp16 ones hide the difference.
template <int V, int H, bool ROUND>
struct Tile {
    static constexpr int NT = 64 * H;
    static constexpr int VB = V / 8;
    static constexpr int kStages = H == 2 ? 3 : 4;                  // steps in the ring: one in work, the others in flight
    static constexpr int kRowBytes = NT * 2;
    static constexpr int kStageBytes = kStep * kRowBytes + kStep * V * 2;
    static constexpr int kPitch = NT + 4;                           // floats per row of the tile of sums (conflict-free)
    static constexpr int kSumBytes = V * kPitch * 4;
    // shared memory of one warp: the ring of steps, later the warp's tile of sums
    static constexpr int kWarpBytes = kStages * kStageBytes > kSumBytes ? kStages * kStageBytes : kSumBytes;
    static constexpr int kPieces = NT / 8;                          // eight-column pieces of a row of C
    static constexpr int kUnits = V * kPieces / 32;                 // a unit: one piece per lane
    static constexpr int kFloats = V * NT;
    float acc[VB][4 * H][4];                                        // [rows 8 vb ..][columns 16 x ..][one instruction's]

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int vb = 0; vb < VB; ++vb)
#pragma unroll
            for (int x = 0; x < 4 * H; ++x)
#pragma unroll
                for (int d = 0; d < 4; ++d) acc[vb][x][d] = 0.f;
    }
    __device__ __forceinline__ void mma(int x, const uint32_t (&a)[4], const uint32_t (&b)[VB][2]) {
#pragma unroll
        for (int vb = 0; vb < VB; ++vb) {
            if constexpr (ROUND) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                mma_16816(d, a[0], a[1], a[2], a[3], b[vb][0], b[vb][1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[vb][x][e] += d[e];
            } else {
                mma_16816(acc[vb][x], a[0], a[1], a[2], a[3], b[vb][0], b[vb][1]);
            }
        }
    }
    // Column ids of two steps, one per lane (lanes 0-15 the first step, 16-31 the second); -1 past the end.
    static __device__ __forceinline__ int load_cols(const int* __restrict__ col, int j0, int len, int step, int stride, int lane) {
        const unsigned idx = (unsigned)(step + (lane >> 4) * stride) * kStep + (lane & 15);
        return idx < (unsigned)len ? __ldg(col + j0 + idx) : -1;
    }
    // (The rings have to start on 128-byte boundaries, also behind a kernel's other shared variables: 16 bytes off, a copied row of 128
    // bytes is written in two pieces; 4000 rows of 160 vectors, N = 128, 47 us, 21 as it is.)
    // Rows of the step land as [16 vectors][NT] with their 16-byte pieces XOR-swizzled by the vector number, so that the
    // copies (eight lanes per 128 bytes) and ldmatrix (eight rows per matrix) both touch every bank once.
    static __device__ __forceinline__ void copy_step(const Problem& p, const __half* __restrict__ values, const __half* __restrict__ rhs,
                                                     int n0, int j0, int len, int s, int cols, int half, int lane, uint32_t slot) {
        constexpr int kLanes = kPieces;                     // lanes per row of B
        constexpr int kRows = 32 / kLanes;
        const int piece = lane % kLanes;
        const bool in_n = n0 + piece * 8 < p.ldb;
        const __half* base = rhs + n0 + piece * 8;
#pragma unroll
        for (int i = 0; i < kStep / kRows; ++i) {
            const int r = i * kRows + lane / kLanes;
            const int c = __shfl_sync(0xffffffffu, cols, half * 16 + r);
            const bool ok = in_n && (unsigned)c < (unsigned)p.K;
            cp_async_16(slot + r * kRowBytes + ((piece ^ (r & 7)) << 4), ok ? base + (int64_t)c * p.ldb : rhs, ok);
        }
        const int k = lane / VB, part = lane % VB;
        if (lane < kStep * VB) {
            const unsigned idx = (unsigned)s * kStep + k;
            const bool ok = idx < (unsigned)len;
            cp_async_16(slot + kStep * kRowBytes + k * (V * 2) + ((V == 16 ? part ^ ((k >> 2) & 1) : 0) << 4),
                        ok ? values + ((int64_t)j0 + idx) * V + part * 8 : values, ok);
        }
    }
    __device__ __forceinline__ void multiply_step(uint32_t slot, int lane) { multiply_step(slot, slot + kStep * kRowBytes, lane); }
    __device__ __forceinline__ void multiply_step(uint32_t slot, uint32_t vectors, int lane) {
        uint32_t b[VB][2];
        const int k = lane & 15;
        const uint32_t vrow = vectors + k * (V * 2);
        if constexpr (V == 8) {
            ldmatrix_x2_trans(b[0][0], b[0][1], vrow);
        } else {
            uint32_t r[4];
            ldmatrix_x4_trans(r, vrow + (((lane >> 4) ^ ((k >> 2) & 1)) << 4));
            b[0][0] = r[0]; b[0][1] = r[1]; b[VB - 1][0] = r[2]; b[VB - 1][1] = r[3];
        }
        const int kr = (lane >> 4) * 8 + (lane & 7), odd = (lane >> 3) & 1;
        const uint32_t row = slot + kr * kRowBytes;
#pragma unroll
        for (int x = 0; x < 4 * H; ++x) {
            uint32_t a[4];
            ldmatrix_x4_trans(a, row + (((2 * x + odd) ^ (kr & 7)) << 4));
            mma(x, a, b);
        }
    }
    // Adds steps first, first + stride, ... of vectors [j0, j0 + len).  The whole warp takes part; `mem` is its shared memory.
    __device__ __forceinline__ void accumulate(const Problem& p, const __half* __restrict__ values, const __half* __restrict__ rhs, int n0,
                                               int j0, int len, int first, int stride, int lane, uint32_t mem) {
        const int steps = (int)(((unsigned)len + kStep - 1) / kStep);
        if (first >= steps) return;
        const int mine = (steps - first + stride - 1) / stride;         // steps of this warp
        int cols = load_cols(p.col, j0, len, first, stride, lane);
        int next = load_cols(p.col, j0, len, first + 2 * stride, stride, lane);
        int issued = 0;
        uint32_t fill = 0, use = 0;                                     // ring slots
        auto issue = [&]() {
            if (issued < mine)
                copy_step(p, values, rhs, n0, j0, len, first + issued * stride, cols, issued & 1, lane, mem + fill * kStageBytes);
            cp_async_commit();
            if (issued & 1) {
                cols = next;
                next = load_cols(p.col, j0, len, first + (issued + 3) * stride, stride, lane);
            }
            ++issued;
            fill = fill + 1 == kStages ? 0 : fill + 1;
        };
#pragma unroll
        for (int k = 0; k < kStages - 1; ++k) issue();
        for (int k = 0; k < mine; ++k) {
            cp_async_wait<kStages - 2>();
            __syncwarp();                           // everyone's copies are in, and the slot refilled next has been read
            issue();
            multiply_step(mem + use * kStageBytes, lane);
            use = use + 1 == kStages ? 0 : use + 1;
        }
        cp_async_wait<0>();
        __syncwarp();                               // the ring may be used for something else
    }
    // The same from a B whose rows start anywhere (pitch p.ldb halfs, B itself on a 16-byte boundary and of less than 2 GiB), 64 columns: the
    // aligned pieces that hold a row's columns land as they lie, nine per row, and a step's rows are shifted into place before it is
    // multiplied, each piece by the lane that asked for it.  Nothing is read past a row's columns.
    static constexpr int kRawRow = 9 * 16;
    static constexpr int kRawStage = kStep * kRawRow + kStep * V * 2;                          // rows, vectors
    static constexpr int kRawStages = 4;
    static constexpr int kRawBytes = kStep * kRowBytes + kRawStages * kRawStage;               // a step's shifted rows, the ring
    static constexpr int kRawWarpBytes = ((kRawBytes > kSumBytes ? kRawBytes : kSumBytes) + 127) & ~127;
    __device__ __forceinline__ void accumulate_unaligned(const Problem& p, const __half* __restrict__ values, const __half* __restrict__ rhs, int n0,
                                                         int j0, int len, int first, int stride, int lane, uint32_t mem) {
        static_assert(H == 1 && kRawStages == 4, "eight pieces per row; the offsets of four steps in 64 bits");
        const int steps = (int)(((unsigned)len + kStep - 1) / kStep);
        if (first >= steps) return;
        const int mine = (steps - first + stride - 1) / stride;
        const int width = min(NT, p.ldb - n0) * 2, pitch = p.ldb * 2, at0 = n0 * 2;
        const uint8_t* const base = reinterpret_cast<const uint8_t*>(rhs);
        const uint32_t ring = mem + kStep * kRowBytes;
        const int row = lane >> 3, piece = lane & 7;
        int cols = load_cols(p.col, j0, len, first, stride, lane);
        int next = load_cols(p.col, j0, len, first + 2 * stride, stride, lane);
        int issued = 0;
        uint32_t fill = ring, use = ring;
        uint64_t offsets = 0;                       // of this lane's four rows, 4 bits each, of the last four steps asked for
        auto issue = [&]() {
            offsets >>= 16;
            if (issued < mine) {
                const int half = (issued & 1) * 16;
                uint32_t mask = 0;
#pragma unroll
                for (int i = 0; i < 5; ++i) {       // four rows at a time; then the ninth pieces of all
                    const int r = i < 4 ? i * 4 + row : lane & 15, x = i < 4 ? piece : 8;
                    const int c = __shfl_sync(0xffffffffu, cols, half + r);
                    const bool ok = (unsigned)c < (unsigned)p.K;
                    const int at = c * pitch + at0, from = (at & ~15) + x * 16;
                    const int bytes = ok ? min(max(at + width - from, 0), 16) : 0;
                    if (i < 4 || lane < 16) cp_async_bytes(fill + r * kRawRow + x * 16, base + (bytes ? from : 0), (uint32_t)bytes);
                    if (i < 4) mask |= (uint32_t)(at & 15) << (4 * i);
                }
                offsets |= (uint64_t)mask << 48;
                const int k = lane / VB, part = lane % VB;
                if (lane < kStep * VB) {
                    const unsigned idx = (unsigned)(first + issued * stride) * kStep + k;
                    const bool ok = idx < (unsigned)len;
                    cp_async_16(fill + kStep * kRawRow + k * (V * 2) + ((V == 16 ? part ^ ((k >> 2) & 1) : 0) << 4),
                                ok ? values + ((int64_t)j0 + idx) * V + part * 8 : values, ok);
                }
            }
            cp_async_commit();
            if (issued & 1) {
                cols = next;
                next = load_cols(p.col, j0, len, first + (issued + 3) * stride, stride, lane);
            }
            ++issued;
            fill = fill == ring + (kRawStages - 1) * kRawStage ? ring : fill + kRawStage;
        };
#pragma unroll
        for (int k = 0; k < kRawStages - 1; ++k) issue();
        for (int k = 0; k < mine; ++k) {
            cp_async_wait<kRawStages - 2>();
            __syncwarp();                           // everyone's copies are in; the slot refilled next and the shifted rows have been read
            issue();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = i * 4 + row;
                const uint32_t by = (uint32_t)offsets >> (4 * i), at = use + r * kRawRow + piece * 16 + (by & 8);
                uint32_t w[6];
#pragma unroll
                for (int x = 0; x < 6; x += 2) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[x]), "=r"(w[x + 1]) : "r"(at + x * 4) : "memory");
#pragma unroll
                for (int x = 0; x < 5; ++x) w[x] = (by & 4) ? w[x + 1] : w[x];
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = __funnelshift_r(w[x], w[x + 1], (by & 2) * 8);
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(mem + r * kRowBytes + ((piece ^ (r & 7)) << 4)), "r"(w[0]), "r"(w[1]),
                             "r"(w[2]), "r"(w[3]) : "memory");
            }
            __syncwarp();                           // the step's rows are in place
            multiply_step(mem, use + kStep * kRawRow, lane);
            use = use == ring + (kRawStages - 1) * kRawStage ? ring : use + kRawStage;
        }
        cp_async_wait<0>();
        __syncwarp();
    }
    // This warp's accumulators to its tile of sums [V][kPitch].
    __device__ __forceinline__ void spill(float* dst, int lane) const {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int vb = 0; vb < VB; ++vb)
#pragma unroll
            for (int x = 0; x < 4 * H; ++x)
#pragma unroll
                for (int d = 0; d < 4; ++d)
                    dst[(vb * 8 + 2 * t + (d & 1)) * kPitch + 16 * x + g + 8 * (d >> 1)] = acc[vb][x][d];
    }
    // This lane's piece of unit u in a tile of sums.
    static __device__ __forceinline__ int piece_at(int u, int lane) {
        const int id = u * 32 + lane;
        return (id / kPieces) * kPitch + (id % kPieces) * 8;
    }
    static __device__ __forceinline__ void add_piece(const float* src, float (&o)[8]) {
        const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
        o[0] += lo.x; o[1] += lo.y; o[2] += lo.z; o[3] += lo.w;
        o[4] += hi.x; o[5] += hi.y; o[6] += hi.z; o[7] += hi.w;
    }
    // Writes this lane's piece of unit u to C (first_row: the first of the vector row's V rows).
    template <typename OutT, bool ADD = false>
    static __device__ __forceinline__ void store_unit(const Problem& p, OutT* __restrict__ out, int64_t first_row, int n0, int u, int lane,
                                                      float (&o)[8], const __half* add = nullptr) {
        const int id = u * 32 + lane, n = n0 + (id % kPieces) * 8;
        if (p.bias) {
            const float b = __half2float(p.bias[first_row + id / kPieces]);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] += b;
        }
        if (ADD && add && n < p.N) {                             // (rows are whole pieces)
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(add + (first_row + id / kPieces) * p.N + n));
            const uint32_t x[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&x[e]));
                o[2 * e] += f.x; o[2 * e + 1] += f.y;
            }
        }
        OutT* dst = out + (first_row + id / kPieces) * p.N + n;
        if (p.out_pieces) {
            if (n >= p.N) return;                                // rows of C are whole pieces: all eight or none
            if constexpr (sizeof(OutT) == 2) {
                const __half2 h0 = __floats2half2_rn(o[0], o[1]), h1 = __floats2half2_rn(o[2], o[3]);
                const __half2 h2 = __floats2half2_rn(o[4], o[5]), h3 = __floats2half2_rn(o[6], o[7]);
                uint4 w;
                w.x = *reinterpret_cast<const uint32_t*>(&h0); w.y = *reinterpret_cast<const uint32_t*>(&h1);
                w.z = *reinterpret_cast<const uint32_t*>(&h2); w.w = *reinterpret_cast<const uint32_t*>(&h3);
                *reinterpret_cast<uint4*>(dst) = w;
            } else {
                *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<float4*>(dst + 4) = make_float4(o[4], o[5], o[6], o[7]);
            }
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (n + e < p.N) {
                    if constexpr (sizeof(OutT) == 2) dst[e] = __float2half_rn(o[e]);
                    else dst[e] = o[e];
                }
        }
    }
    // Four columns of one row to C.
    template <typename OutT>
    static __device__ __forceinline__ void store_four(const Problem& p, OutT* __restrict__ out, int64_t row, int n, float4 o) {
        OutT* dst = out + row * p.N + n;
        if (p.bias) {
            const float b = __half2float(p.bias[row]);
            o.x += b; o.y += b; o.z += b; o.w += b;
        }
        if (p.out_pieces) {
            if (n >= p.N) return;
            if constexpr (sizeof(OutT) == 2) {
                const __half2 h0 = __floats2half2_rn(o.x, o.y), h1 = __floats2half2_rn(o.z, o.w);
                *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            } else {
                *reinterpret_cast<float4*>(dst) = o;
            }
        } else {
            const float v[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < p.N) {
                    if constexpr (sizeof(OutT) == 2) dst[e] = __float2half_rn(v[e]);
                    else dst[e] = v[e];
                }
        }
    }
    // A warp's own tile to C, eight rows at a time through one slot of its ring.
    template <typename OutT, bool ADD = false>
    __device__ __forceinline__ void store(const Problem& p, OutT* __restrict__ out, int64_t first_row, int n0, float* slot, int lane,
                                          const __half* add = nullptr) const {
        static_assert(8 * kPitch * 4 <= kWarpBytes, "eight rows of sums fit the ring");
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int vb = 0; vb < VB; ++vb) {
#pragma unroll
            for (int x = 0; x < 4 * H; ++x)
#pragma unroll
                for (int d = 0; d < 4; ++d) slot[(2 * t + (d & 1)) * kPitch + 16 * x + g + 8 * (d >> 1)] = acc[vb][x][d];
            __syncwarp();
#pragma unroll
            for (int u = 0; u < kUnits / VB; ++u) {
                float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                add_piece(slot + piece_at(u, lane), o);
                store_unit<OutT, ADD>(p, out, first_row + vb * 8, n0, u, lane, o, add);
            }
            __syncwarp();
        }
    }
};

// One launch, no scratch: an item (vector row, column tile, batch entry) is done by `team` warps of a CTA (1, 2, 4 or 8)
// or, with clusters, by all warps of `cluster` CTAs; the warps take 16-vector steps in turn and their sums are added in
// warp order through shared memory (of the cluster), so results do not depend on timing.
// cta_item: the first of the CTA's (or cluster's) items, of problem p.  (With the warp's own item in its place the plain kernel of V = 16
// took another register and 2 to 5 % more time: 2048 x 4608 at 90 %, N = 2048 225 us, 216 as it is; 1500 x 2500 at 80 %, N = 800 60.3 and 57.0.)
template <int V, typename OutT, int H, bool ADD = false, bool UNALIGNED = false>
__device__ __forceinline__ void do_items(const Problem& p, OutT* __restrict__ out, long long cta_item, int team, int cluster,
                                         const __half* add = nullptr) {
    using T = Tile<V, H, sizeof(OutT) == 4>;
    constexpr int kMine = UNALIGNED ? T::kRawWarpBytes : T::kWarpBytes;
    extern __shared__ __align__(128) uint8_t smem[];    // [warp][kMine]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = cluster > 1 ? (int)cluster_cta_rank() : 0;
    const int member = warp % team;
    const Where w = locate(p, cta_item + warp / team, T::NT);
    uint8_t* const mem = smem + warp * kMine;
    T tile;
    tile.clear();
    if (w.row >= 0) {
        if constexpr (UNALIGNED)
            tile.accumulate_unaligned(p, p.values, p.rhs, w.n0, w.j0, w.len, rank * team + member, team * cluster, lane, smem_u32(mem));
        else
            tile.accumulate(p, p.values + w.batch * p.values_stride, p.rhs + w.batch * p.rhs_stride, w.n0, w.j0, w.len, rank * team + member,
                            team * cluster, lane, smem_u32(mem));
    }
    OutT* const cbase = out + w.batch * p.out_stride;
    const int64_t first_row = (int64_t)w.row * V;
    if (team == 1) {
        if (w.row >= 0) tile.template store<OutT, ADD>(p, cbase, first_row, w.n0, reinterpret_cast<float*>(mem), lane, add);
        return;
    }
    tile.spill(reinterpret_cast<float*>(mem), lane);
    __syncthreads();
    static_assert(T::kUnits <= kWarps && T::kFloats * 4 <= kWarps * T::kWarpBytes, "one unit per warp");
    float kept[8];
    for (int u = member; u < T::kUnits; u += team) {
        float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int m = 0; m < team; ++m)
            T::add_piece(reinterpret_cast<const float*>(smem + (warp - member + m) * kMine) + T::piece_at(u, lane), o);
        if (cluster == 1) {
            if (w.row >= 0) T::template store_unit<OutT, ADD>(p, cbase, first_row, w.n0, u, lane, o, add);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) kept[e] = o[e];
        }
    }
    if (cluster == 1) return;
    __syncthreads();                                      // the warps' tiles are read: the CTA's tile takes their place
    float* const whole = reinterpret_cast<float*>(smem);
    if (warp < T::kUnits)
#pragma unroll
        for (int e = 0; e < 8; ++e) whole[(warp * 8 + e) * 32 + lane] = kept[e];
    cluster_sync_all();                                   // every CTA's tile is complete and visible
    for (int u = warp; u < T::kUnits; u += kWarps) {
        if (u % cluster != rank) continue;                // the units are dealt over the CTAs
        float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const uint32_t at = smem_u32(whole + u * 256 + lane);
        for (int c = 0; c < cluster; ++c) {
            const uint32_t remote = cluster_map_shared(at, (uint32_t)c);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] += ld_cluster_f32(remote + e * 128);
        }
        if (w.row >= 0) T::template store_unit<OutT, ADD>(p, cbase, first_row, w.n0, u, lane, o, add);
    }
    cluster_sync_all();                                   // nobody leaves while its tile is being read
}

template <int V, typename OutT, int H>
__global__ void __launch_bounds__(kThreads, kResident)
sspmm_rows_kernel(const __grid_constant__ Problem p, OutT* __restrict__ out, int team, int cluster) {
    do_items<V, OutT, H>(p, out, (long long)(blockIdx.x / cluster) * (kWarps / team), team, cluster);
}

// A dense operand whose rows start off 16-byte boundaries, read where it lies: the aligned copy is an allocation and a launch of its own.
// 512 x 512 half full, V = 8, N = 49 9.8 us with the copy, 6.2 here (replayed from a graph 5.1 and 4.3); 512 x 4608 at 80 % 12.3 and 8.7 (7.1, 6.8).  A step costs
// more than twice an aligned one, in shared memory: its rows are read from the ring, shifted and written once more.
template <int V, typename OutT>
__global__ void __launch_bounds__(kThreads, kResident)
sspmm_rows_unaligned_kernel(const __grid_constant__ Problem p, OutT* __restrict__ out, int team, int cluster) {
    do_items<V, OutT, 1, false, true>(p, out, (long long)(blockIdx.x / cluster) * (kWarps / team), team, cluster);
}

// Few items, and a row of unknown length may be many times the mean: a cluster has up to sixteen items, and its 64 warps take them in numbers that
// go with their steps (per_step warps each, 16 bits of fraction).  What does not fit the warps at once is done in another round;
// even rows fit.  A row's warps depend on its own length alone, so results do not depend on the order of the rows.
// One launch without scratch, where cutting such rows (below) is a list by one CTA and a launch that waits for it, and leaves
// one warp to a row of 256 vectors: 128 rows of 230 of 4608, V = 8, N = 49 17 us, here 8.2; one of them full 15.2, 10.3; 32 rows of 115 of
// 2304, N = 800 16.7, 8.2.  What bounds it are the chain of look-ups, a step or two, and the cluster's start and two barriers.
// The items are dealt in turn and staggered, so that tiles of one row do not meet (32 rows, one full, N = 800: 20.5 us in plain
// turns, 10.3).
constexpr int kStagger = 113;
constexpr int kPooled = 16;               // items per cluster
constexpr int kPoolClusters = 32;         // all of them resident
constexpr int kPoolWarps = kMaxCluster * kWarps;
constexpr int kPoolMost = 40;             // warps of an item, so that others find room (all 64: 128 rows of 115, one full, 16.4 us, 10.3)
template <int V, typename OutT, int H>
__global__ void __launch_bounds__(kThreads, kResident)
sspmm_rows_pooled_kernel(const __grid_constant__ Problem p, OutT* __restrict__ out, int per_step, int most) {
    using T = Tile<V, H, sizeof(OutT) == 4>;
    extern __shared__ __align__(128) uint8_t smem[];    // [warp][T::kWarpBytes]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mine = (int)cluster_cta_rank() * kWarps + warp;
    const int clusters = gridDim.x / kMaxCluster, id = blockIdx.x / kMaxCluster;
    const int count = (int)((p.items + clusters - 1) / clusters);
    // Every lane has one item, whose warps end before `end` (of the warps of all items, one after another).
    Where own = {-1, 0, 0, 0, 0};
    if (lane < count) own = locate(p, (long long)lane * clusters + (id + lane * kStagger) % clusters, T::NT);
    const int steps = (int)(((unsigned)own.len + kStep - 1) / kStep);
    const int share = own.row < 0 ? 0 : min(max((int)((long long)steps * per_step >> 16), 1), most);
    int end = share;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += below;
    }
    uint8_t* const mem = smem + warp * T::kWarpBytes;
    const int all = __shfl_sync(0xffffffffu, end, 31);
    for (int done = 0; done < all;) {                     // a round: the items that fit from here on (the same in every warp)
        const unsigned fits = __ballot_sync(0xffffffffu, end > done && end <= done + kPoolWarps);
        const unsigned before = __ballot_sync(0xffffffffu, end - share <= done + mine);
        const int owner = 31 - __clz(before);             // (of items without warps the last, whose end is the same)
        const int last = __shfl_sync(0xffffffffu, end, 31 - __clz(fits));
        const int team = __shfl_sync(0xffffffffu, share, owner), first = __shfl_sync(0xffffffffu, end, owner) - team - done;
        const int row = __shfl_sync(0xffffffffu, own.row, owner), n0 = __shfl_sync(0xffffffffu, own.n0, owner);
        const int j0 = __shfl_sync(0xffffffffu, own.j0, owner), len = __shfl_sync(0xffffffffu, own.len, owner);
        const bool works = done + mine < last;
        const int64_t first_row = (int64_t)row * V;
        if (works) {
            T tile;
            tile.clear();
            tile.accumulate(p, p.values, p.rhs, n0, j0, len, mine - first, team, lane, smem_u32(mem));
            if (team == 1) tile.store(p, out, first_row, n0, reinterpret_cast<float*>(mem), lane);
            else tile.spill(reinterpret_cast<float*>(mem), lane);
        }
        cluster_sync_all();                               // every warp's tile is complete and visible
        if (works && team > 1) {
            constexpr int kFours = T::NT / 4;
            for (int u = mine - first; u < V * kFours / 32; u += team) {
                const int x = u * 32 + lane, r = x / kFours, n = x % kFours * 4;
                const uint32_t piece = smem_u32(smem) + (r * T::kPitch + n) * 4;
                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
                for (int m = first; m < first + team; ++m) {
                    const float4 v = ld_cluster_f32x4(cluster_map_shared(piece + m % kWarps * T::kWarpBytes, (uint32_t)(m / kWarps)));
                    o.x += v.x; o.y += v.y; o.z += v.z; o.w += v.w;
                }
                T::store_four(p, out, first_row + r, n0 + n, o);
            }
        }
        cluster_sync_all();                               // the tiles have been read: the rings may be used again, and a CTA may leave
        done = last;
    }
}

// More items than warps, one warp each: a CTA has its share of the items from the start, looks all of them up at once (a thread each, the
// first column ids on their way to L1), and its warps take them one after another from a counter in shared memory.  With a CTA for
// every eight items the look-ups, four dependent loads, were paid for by every round of CTAs, and a warp that was done waited for
// the longest of its eight rows.  96 products of 512 x 512 at 90 %, N = 64: 12.5 us, now 10.5.
// Nothing is known of the rows' lengths here, so nothing is dealt to a warp ahead of time: with the items dealt to the warps in turn and
// the next two looked up early, one row in a hundred of 512 vectors among rows of 5 took 32 us where the CTAs of eight took 19 (now
// 15); what look-ups are left, half a microsecond a launch, shows with rows of ten vectors (7.7 us, dealt in turn 7.1).
// The CTAs' shares are staggered: rows are often ordered by length, and their number may divide the number of CTAs.
// (Vectors of 16 rows do not gain: 96 products of 512 x 512 at 90 %, N = 64 8.3 us, walking 8.6; 1355 x 4242, N = 16200 192 and 217.)
template <typename OutT, int H>
__global__ void __launch_bounds__(kThreads, kResident)
sspmm_rows_walk_kernel(const __grid_constant__ Problem p, OutT* __restrict__ out) {
    constexpr int V = 8;
    using T = Tile<V, H, sizeof(OutT) == 4>;
    extern __shared__ __align__(128) uint8_t smem[];    // [warp][T::kWarpBytes]
    __shared__ Where table[kThreads];
    __shared__ int next;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* const mem = smem + warp * T::kWarpBytes;
    const long long rounds = (p.items + gridDim.x - 1) / gridDim.x;
    for (long long r0 = 0; r0 < rounds; r0 += kThreads) {
        const long long r = r0 + threadIdx.x;
        if (r0 > 0) __syncthreads();                     // the table has been read
        if (r < rounds) {
            const Where w = locate(p, r * gridDim.x + (blockIdx.x + r * kStagger) % gridDim.x, T::NT);
            if (w.len > 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(p.col + w.j0));
            table[threadIdx.x] = w;
        }
        if (threadIdx.x == 0) next = 0;
        __syncthreads();
        const int count = (int)min((long long)kThreads, rounds - r0);
        for (;;) {
            int x = 0;
            if (lane == 0) x = atomicAdd(&next, 1);
            x = __shfl_sync(0xffffffffu, x, 0);
            if (x >= count) break;
            const Where w = table[x];
            if (w.row < 0) continue;
            T tile;
            tile.clear();
            tile.accumulate(p, p.values + w.batch * p.values_stride, p.rhs + w.batch * p.rhs_stride, w.n0, w.j0, w.len, 0, 1, lane, smem_u32(mem));
            tile.store(p, out + w.batch * p.out_stride, (int64_t)w.row * V, w.n0, reinterpret_cast<float*>(mem), lane);
        }
    }
}

// Several products in one launch: the items of one after those of the other.
// The four launches of an encoder layer at 1 x 128 tokens (32 to 128 CTAs of 256 threads)
// take 5.8 to 7.9 us each from cold caches.
struct ProblemSet {
    int count;
    int first[kRowsMaxSet + 1];           // first item of each product, and the end
    void* out[kRowsMaxSet];
    const __half* add[kRowsMaxSet];       // like C, added to the sums; or null (only looked at with ADD)
    Problem p[kRowsMaxSet];
};
template <int V, typename OutT, int H, bool ADD>
__global__ void __launch_bounds__(kThreads, kResident)
sspmm_rows_set_kernel(const __grid_constant__ ProblemSet s, int team, int cluster) {
    const int per_cta = kWarps / team, warp = threadIdx.x >> 5;
    const long long item = (long long)(blockIdx.x / cluster) * per_cta + warp / team;
    int k = 0;
    while (k + 1 < s.count && item >= s.first[k + 1]) ++k;
    do_items<V, OutT, H, ADD>(s.p[k], static_cast<OutT*>(s.out[k]), item - warp / team - s.first[k], team, cluster,
                            ADD ? s.add[k] : nullptr);
}

// Matrices whose rows differ in length by orders of magnitude (power-law matrices: half of the rows have fewer than 50
// vectors, the longest tens of thousands; n = 51970, V = 8, N = 128: 40.8 us, with one CTA of tcgen05 stages per SM 67.8).
// Rows longer than kLightRow are cut into parts of at most p.chunk vectors (listed by list_parts_kernel); a CTA does a
// part with all its warps, the parts dealt out in turn since they are of one size, and whoever finishes the last part of
// a row adds the parts up in order.  Rows of a single part follow those with several: they write C themselves and have no
// partial sums.  Then the warps, each on its own, take the remaining rows in the caller's order from a counter.
template <int V, typename OutT, int H>
__global__ void __launch_bounds__(kThreads, kResident)
sspmm_rows_split_kernel(const __grid_constant__ Problem p, OutT* __restrict__ out) {
    using T = Tile<V, H, sizeof(OutT) == 4>;
    extern __shared__ __align__(128) uint8_t smem[];    // [warp][T::kWarpBytes]
    __shared__ int seen;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* const mem = smem + warp * T::kWarpBytes;
    // The list was sized from a vector count; if the matrix needs more parts than fit, nothing is cut.
    const int several = p.header[0], whole = p.header[2];
    const bool cut = several <= p.cap_cut && whole <= p.cap_whole;
    const int parts_total = cut ? (several + whole) * p.n_tiles : 0;
    const int none = INT_MAX;
    auto entry = [&](int at) {
        const int i = at / p.n_tiles;
        return p.entries[i < several ? i : p.cap_cut + (i - several)];
    };
    int x = (int)blockIdx.x < parts_total ? (int)blockIdx.x : none;
    int4 en = x < parts_total ? entry(x) : make_int4(0, 0, 0, 0);
    while (x < parts_total) {
        const int x2 = x < parts_total - (int)gridDim.x ? x + (int)gridDim.x : none;
        int4 en2 = make_int4(0, 0, 0, 0);
        if (x2 < parts_total) en2 = entry(x2);
        const int nt = x % p.n_tiles, part = en.w & 0xffff, parts = (int)((unsigned)en.w >> 16);
        T tile;
        tile.clear();
        tile.accumulate(p, p.values, p.rhs, nt * T::NT, en.y, en.z, warp, kWarps, lane, smem_u32(mem));
        tile.spill(reinterpret_cast<float*>(mem), lane);
        __syncthreads();
        const int first = x - part * p.n_tiles;                          // the row's part 0 for this column tile
        for (int u = warp; u < T::kUnits; u += kWarps) {
            float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int m = 0; m < kWarps; ++m)
                T::add_piece(reinterpret_cast<const float*>(smem + m * T::kWarpBytes) + T::piece_at(u, lane), o);
            if (parts == 1) {
                T::store_unit(p, out, (int64_t)en.x * V, nt * T::NT, u, lane, o);
            } else {
                float4* dst = reinterpret_cast<float4*>(p.partial + (int64_t)x * T::kFloats) + u * 64 + lane * 2;
                __stcg(dst, make_float4(o[0], o[1], o[2], o[3]));
                __stcg(dst + 1, make_float4(o[4], o[5], o[6], o[7]));
            }
        }
        if (parts > 1) {
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) seen = atomicAdd(p.arrivals + first, 1);
            __syncthreads();
            if (seen == parts - 1) {
                // four columns per thread; sixteen parts' loads are under way together
                __threadfence();
                const int64_t step = (int64_t)p.n_tiles * (T::kFloats / 4);
                for (int f = threadIdx.x; f < T::kFloats / 4; f += kThreads) {
                    const float4* src = reinterpret_cast<const float4*>(p.partial + (int64_t)first * T::kFloats) + f;
                    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int c0 = 0; c0 < parts; c0 += 16) {
                        float4 v[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c)
                            v[c] = c0 + c < parts ? __ldcg(src + (c0 + c) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int c = 0; c < 16; ++c) { o.x += v[c].x; o.y += v[c].y; o.z += v[c].z; o.w += v[c].w; }
                    }
                    T::store_four(p, out, (int64_t)en.x * V + f * 4 / T::NT, nt * T::NT + f * 4 % T::NT, o);
                }
            }
        }
        __syncthreads();                                  // the tiles of sums and `seen` are free again
        x = x2; en = en2;
    }
    // row items, one warp each; the next item is looked up while the current one is in work
    auto take = [&]() {
        int T0 = 0;
        if (lane == 0) T0 = atomicAdd(p.header + 1, 1);
        return (long long)__shfl_sync(0xffffffffu, T0, 0);
    };
    long long at = take();
    Where w = locate(p, at, T::NT);
    while (at < p.items) {
        const long long at2 = take();
        const Where w2 = locate(p, at2, T::NT);
        if (w.row >= 0 && !(cut && w.len > kLightRow)) {
            T tile;
            tile.clear();
            tile.accumulate(p, p.values, p.rhs, w.n0, w.j0, w.len, 0, 1, lane, smem_u32(mem));
            tile.store(p, out, (int64_t)w.row * V, w.n0, reinterpret_cast<float*>(mem), lane);
        }
        at = at2; w = w2;
    }
}

// The list of parts (the parts of a row are consecutive, part 0 first), cleared arrival counters and, with one CTA, the
// header; with several the header is zero at launch.
__global__ void __launch_bounds__(1024)
list_parts_kernel(const __grid_constant__ Problem p) {
    __shared__ int count[2];
    const bool alone = gridDim.x == 1;
    if (threadIdx.x < 2) count[threadIdx.x] = 0;
    __syncthreads();
    const int stride = gridDim.x * 1024;
    for (int x = blockIdx.x * 1024 + threadIdx.x; x < p.cap_cut * p.n_tiles; x += stride) p.arrivals[x] = 0;
    for (int64_t b = blockIdx.x * 1024 + threadIdx.x; b < p.m_vec; b += 4LL * stride) {
        int j0[4], len[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t i = b + (int64_t)k * stride;
            j0[k] = i < p.m_vec ? __ldg(p.row_offsets + i) : 0;
            len[k] = i < p.m_vec ? __ldg(p.row_offsets + i + 1) - j0[k] : 0;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (len[k] <= kLightRow) continue;
            const int row = (int)(b + (int64_t)k * stride);
            if (len[k] <= p.chunk) {
                const int at = alone ? atomicAdd(&count[1], 1) : atomicAdd(p.header + 2, 1);
                if (at < p.cap_whole) p.entries[p.cap_cut + at] = make_int4(row, j0[k], len[k], 1 << 16);
                continue;
            }
            const int n = (int)(((unsigned)len[k] + p.chunk - 1) / p.chunk);
            const int first = alone ? atomicAdd(&count[0], n) : atomicAdd(p.header, n);
            for (int c = 0; c < n && first + c < p.cap_cut; ++c)
                p.entries[first + c] = make_int4(row, j0[k] + c * p.chunk, min(p.chunk, len[k] - c * p.chunk), n << 16 | c);
        }
    }
    __syncthreads();
    if (alone && threadIdx.x == 0) { p.header[0] = count[0]; p.header[1] = 0; p.header[2] = count[1]; }
}

// How the one-launch kernel divides a product by the mean row.  Tile width: 128 columns halve the work per gathered byte
// outside the loads; 64 when that is all there is or when wide tiles, a CTA each, would leave SMs without one.  Warps per item:
// enough to fill the SMs, at least one step each; long rows get a whole CTA so that no single warp runs long after the others.
struct Division { int H, team, cluster; };
long long count_items(const SpmmArgs* a, int count, int H) {
    long long n = 0;
    for (int k = 0; k < count; ++k) n += (long long)a[k].m_vec * a[k].batch * ((a[k].N + 64 * H - 1) / (64 * H));
    return n;
}
// nvec: vectors of all products (<= 0: unknown)
Division divide(const SpmmArgs* a, int count, long long nvec, int sms) {
    const long long slots = (long long)sms * kResident * kWarps;
    long long rows = 0;
    int widest = 0;
    for (int k = 0; k < count; ++k) { rows += a[k].m_vec; widest = std::max(widest, a[k].N); }
    const long long mean_steps = nvec > 0 ? (nvec / rows + kStep) / kStep : (a->K / 2 + kStep) / kStep;
    Division d{widest > 64 ? 2 : 1, 1, 1};
    if (d.H == 2 && count_items(a, count, 2) * std::min<long long>(mean_steps, kWarps) < slots) d.H = 1;
    const long long want = std::min(slots / count_items(a, count, d.H), mean_steps);
    while (d.team < kWarps && (2 * d.team <= want || mean_steps > 32LL * d.team)) d.team *= 2;
    // Clusters leave each warp fewer steps, at least four, and cost about a microsecond.  The first doubling is not worth it where it gives
    // SMs a second CTA and saves no more than seven steps per warp (300 x 700, V = 8, N = 96 5.34 us in clusters of two, 4.52 without; 512 x 2048,
    // V = 16, N = 200 8.82 and 8.41; 188 x 4491, N = 712, 18 steps saved, 15.2 and 17.0), where a full row leaves no warp more than twenty
    // (64 x 4608, V = 8, N = 1024, one row of eight full: 13.5 us in clusters, 18.5); the second is from two and a half steps on where every
    // CTA has an SM (256 x 1024, V = 16, N = 128 5.34, in clusters of four 4.92; 113 x 1191, V = 16, N = 8 5.17 and 4.63).  fp32 results keep their
    // clusters: their distance from 64 bits grows by 1 to 4 % with other chains (7.74e-8 to 8.04e-8, 336 x 878); fp16 ones show nothing.
    if (d.team == kWarps) {
        const long long items = count_items(a, count, d.H);
        const bool f16 = a->out_f16;
        while (d.cluster < kMaxCluster && (long long)d.cluster * 2 * d.team <= want) {
            const long long warps = (long long)d.cluster * d.team;
            if (f16 && d.cluster == 1 && items <= sms && 2 * items > sms && mean_steps <= 14 * warps && a->K <= 20 * kStep * warps) break;
            if (mean_steps < 4 * warps && !(f16 && d.cluster == 2 && 2 * mean_steps >= 5 * warps && 4 * items <= sms)) break;
            d.cluster *= 2;
        }
    }
    return d;
}

template <typename Kern>
cudaError_t allow_smem(Kern kern, DeviceOnce& once, int bytes) {
    if (once.done()) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (bytes > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) once.mark();
    return e;
}

template <int V, typename OutT, int H, int WARP_BYTES = 0, typename Kern, typename... Args>
cudaError_t launch_items(Kern kern, DeviceOnce& once, long long items, const Division& d, cudaStream_t stream, Args... args) {
    constexpr int kBytes = kWarps * (WARP_BYTES ? WARP_BYTES : Tile<V, H, sizeof(OutT) == 4>::kWarpBytes);
    cudaError_t e = allow_smem(kern, once, kBytes);
    if (e != cudaSuccess) return e;
    const int per_cta = kWarps / d.team;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((items + per_cta - 1) / per_cta * d.cluster));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)kBytes; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)d.cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = d.cluster > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args..., d.team, d.cluster);
}

template <int V, typename OutT, int H>
cudaError_t launch_plain(const SpmmArgs& a, const Problem& p, const Division& d, int sms) {
    if constexpr (V == 8) {
        static DeviceOnce once_walk;
        if (d.team == 1 && p.items > (long long)sms * kResident * kWarps) {
            auto kern = sspmm_rows_walk_kernel<OutT, H>;
            constexpr int kBytes = kWarps * Tile<V, H, sizeof(OutT) == 4>::kWarpBytes;
            const cudaError_t e = allow_smem(kern, once_walk, kBytes);
            if (e != cudaSuccess) return e;
            kern<<<sms * kResident, kThreads, kBytes, a.stream>>>(p, static_cast<OutT*>(a.out));
            return cudaGetLastError();
        }
    }
    static DeviceOnce once;
    return launch_items<V, OutT, H>(sspmm_rows_kernel<V, OutT, H>, once, p.items, d, a.stream, p, static_cast<OutT*>(a.out));
}

template <int V, typename OutT, bool ADD>
cudaError_t launch_set(const ProblemSet& s, const Division& d, cudaStream_t stream) {
    static DeviceOnce once_wide, once_narrow;
    if (d.H == 2) return launch_items<V, OutT, 2>(sspmm_rows_set_kernel<V, OutT, 2, ADD>, once_wide, s.first[s.count], d, stream, s);
    return launch_items<V, OutT, 1>(sspmm_rows_set_kernel<V, OutT, 1, ADD>, once_narrow, s.first[s.count], d, stream, s);
}

template <int V, typename OutT, int H>
cudaError_t launch_split(const SpmmArgs& a, const Problem& p, int sms) {
    auto kern = sspmm_rows_split_kernel<V, OutT, H>;
    constexpr int kBytes = kWarps * Tile<V, H, sizeof(OutT) == 4>::kWarpBytes;
    static DeviceOnce once;
    cudaError_t e = allow_smem(kern, once, kBytes);
    if (e != cudaSuccess) return e;
    const bool alone = a.m_vec <= 16384;                  // one CTA saves the launch that clears the header
    if (!alone) {
        e = cudaMemsetAsync(p.header, 0, 16, a.stream);
        if (e != cudaSuccess) return e;
    }
    list_parts_kernel<<<alone ? 1 : sms, 1024, 0, a.stream>>>(p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    kern<<<sms * kResident, kThreads, kBytes, a.stream>>>(p, static_cast<OutT*>(a.out));
    return cudaGetLastError();
}

// Some row may be many times the mean: the columns bound a row's length, so K tells, and the vector count tells the mean.  Below 2048
// columns that counts only where the plain division leaves a warp more than 48 steps of such a row (a step takes about
// 0.65 us, the list of parts 5): eight rows of 2000 vectors among 1024 of 40, V = 16, N = 128, 41 to 46 us, cut 14; 512 rows of 36 of
// 1200, V = 8, N = 1024, 11 us, listed in vain 15.
// Then, in this order: more warps for every item, warps by length, cut rows.  64 rows of 460 of 4608, V = 8, N = 56: 6.6 us with 32 warps
// per row, 8.2 by length, 10.3 cut; one of them full, 10.3, 10.3 and 16.  Eight rows of 1000 of 20000: 8.2 by length, 12.4 cut, one
// full 14.4 both ways.
struct Route {
    enum Way { kPlain, kPooledWarps, kCut } way;
    Division d;
    bool long_rows;                                 // a row may be many times the mean
    int per_step, most;                             // pooled warps: warps per step of an item (16 bits of fraction), and at most
};
Route route(const SpmmArgs& a, long long nvec, int sms) {
    Route r{Route::kPlain, divide(&a, 1, nvec, sms), false, 0, 0};
    if (nvec <= 0 || a.batch != 1) return r;
    const long long mean = nvec / a.m_vec, slots = (long long)sms * kResident * kWarps, items = count_items(&a, 1, r.d.H);
    if (a.K < 8 * (mean + 1)) return r;
    if (a.K < 2048 && a.K <= 48LL * kStep * r.d.team * r.d.cluster) return r;
    r.long_rows = true;
    // As many warps per item as leave a full row at most twelve steps each, if there is room: a full one then takes no longer than cut.
    Division w = r.d;
    auto too_long = [&] { return a.K > 12LL * kStep * w.team * w.cluster; };
    auto room = [&] { return 2 * items * w.team * w.cluster <= slots; };
    while (too_long() && w.team < kWarps && room()) w.team *= 2;
    while (too_long() && w.cluster < kMaxCluster && w.team == kWarps && room()) w.cluster *= 2;
    if (!too_long()) { r.d = w; return r; }
    // Warps by length, a warp for every two steps at most and so many that even rows take 92 % of them; a full row twelve steps per warp,
    // or twenty where nothing else is in its cluster (eight rows of 1000 of 20000, one full: 14.4 us, and cut).
    const long long pooled = (items + kPoolClusters - 1) / kPoolClusters;
    r.per_step = (int)std::min<long long>(1 << 15, (long long)(0.92 * 65536 * kPoolWarps * kStep * a.m_vec / (pooled * (nvec + 8.0 * a.m_vec))));
    r.most = pooled == 1 ? kPoolWarps : kPoolMost;
    const long long full = std::min<long long>(r.most, std::max<long long>(1, (a.K / kStep * r.per_step) >> 16));
    r.way = pooled <= kPooled && a.K <= (pooled == 1 ? 20 : 12) * kStep * full ? Route::kPooledWarps : Route::kCut;
    return r;
}

template <int V, typename OutT, int H>
cudaError_t launch_pooled(const SpmmArgs& a, const Problem& p, const Route& r) {
    static DeviceOnce once;
    constexpr int kBytes = kWarps * Tile<V, H, sizeof(OutT) == 4>::kWarpBytes;
    cudaError_t e = allow_smem(sspmm_rows_pooled_kernel<V, OutT, H>, once, kBytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(std::min<long long>(p.items, kPoolClusters) * kMaxCluster));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)kBytes; cfg.stream = a.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)kMaxCluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, sspmm_rows_pooled_kernel<V, OutT, H>, p, static_cast<OutT*>(a.out), r.per_step, r.most);
}

template <int V, typename OutT>
cudaError_t launch_typed(const SpmmArgs& a, const Problem& p, int H, const Route& r, int sms) {
    if (r.way == Route::kCut) return H == 2 ? launch_split<V, OutT, 2>(a, p, sms) : launch_split<V, OutT, 1>(a, p, sms);
    if (r.way == Route::kPooledWarps) return H == 2 ? launch_pooled<V, OutT, 2>(a, p, r) : launch_pooled<V, OutT, 1>(a, p, r);
    return H == 2 ? launch_plain<V, OutT, 2>(a, p, r.d, sms) : launch_plain<V, OutT, 1>(a, p, r.d, sms);
}

// Scratch of the variant that cuts rows: [16 B header][cap_cut * n_tiles arrival counters][cap_cut + cap_whole entries]
// [cap_cut * n_tiles partial tiles].
struct Scratch {
    int chunk = 0, cap_cut = 0, cap_whole = 0;      // chunk = 0: not worth cutting
    size_t entries_at = 0, partial_at = 0, bytes = 0;
};
Scratch plan_scratch(const SpmmArgs& a, long long nvec) {
    Scratch r;
    const int sms = current_device_sm_count() > 0 ? current_device_sm_count() : 148;
    if (a.m_vec <= 0 || route(a, nvec, sms).way != Route::kCut) return r;
    const long long nt = a.N <= 64 ? 64 : 128, n_tiles = (a.N + nt - 1) / nt;
    // A part: a quarter of an SM's share of the vectors, at least four steps per warp.  n = 51970 (820 k vectors, V = 8,
    // N = 128) took 46.8 us with a quarter, 52.1 with an eighth and 78 with a sixteenth (every part drains the rings once; measured
    // before the rings were on 128-byte boundaries, 40.8 now).
    long long c = nvec * n_tiles / ((long long)sms * 4) / 128 * 128;
    if (c < 512) c = 512;
    // A row with several parts has at most one that is not full, so its parts are fewer than twice its vectors / c; their
    // partial sums are a few MB at any N (two tiles for each of the sms * 4 shares).
    const long long cap_cut = 2 * nvec / c + 1, cap_whole = nvec / kLightRow + 1;
    const long long tiles = cap_cut * n_tiles, items = tiles + cap_whole * n_tiles;
    if (c > 0x3fffffff || a.K / c >= 32767 || items > 0x3fffffff || tiles * a.V * nt * 4 > (1LL << 30)) return r;
    r.chunk = (int)c; r.cap_cut = (int)cap_cut; r.cap_whole = (int)cap_whole;
    r.entries_at = 16 + (((size_t)tiles * 4 + 15) & ~(size_t)15);
    r.partial_at = r.entries_at + (size_t)(cap_cut + cap_whole) * 16;
    r.bytes = (r.partial_at + (size_t)tiles * a.V * nt * 4 + 255) & ~(size_t)255;
    return r;
}

// Copies [rows][N] (any alignment) to [rows][ld], ld a multiple of 8, zeros in the columns added: one 16-byte piece of
// the copy per thread.
__global__ void __launch_bounds__(256)
align_rows_kernel(const __half* __restrict__ src, __half* __restrict__ dst, int K, int N, int ld, int batch, int64_t src_stride) {
    const int pieces = ld / 8;
    const int64_t total = (int64_t)K * batch * pieces;
    for (int64_t x = (int64_t)blockIdx.x * 256 + threadIdx.x; x < total; x += (int64_t)gridDim.x * 256) {
        const int64_t r = x / pieces;
        const int n = (int)(x - r * pieces) * 8;
        const int64_t b = r / K;
        const unsigned short* s = reinterpret_cast<const unsigned short*>(src + b * src_stride + (r - b * K) * N) + n;
        unsigned short h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) h[e] = n + e < N ? __ldg(s + e) : (unsigned short)0;
        uint4 w;
        w.x = h[0] | (uint32_t)h[1] << 16; w.y = h[2] | (uint32_t)h[3] << 16;
        w.z = h[4] | (uint32_t)h[5] << 16; w.w = h[6] | (uint32_t)h[7] << 16;
        *reinterpret_cast<uint4*>(dst + x * 8) = w;
    }
}

}  // namespace rows

size_t sspmm_rows_scratch_bytes(const SpmmArgs& a, long long nvec) { return rows::plan_scratch(a, nvec).bytes; }

namespace rows {
Problem problem_of(const SpmmArgs& a, int H) {
    Problem p = {};
    p.m_vec = a.m_vec; p.N = a.n_out; p.ldb = a.N; p.K = a.K;
    p.row_indices = a.row_indices; p.row_offsets = a.row_offsets; p.col = a.column_indices;
    p.values = a.values; p.rhs = a.rhs; p.bias = a.bias;
    p.values_stride = a.values_stride; p.rhs_stride = a.rhs_stride; p.out_stride = a.out_stride;
    const size_t es = a.out_f16 ? 2 : 4;
    p.out_pieces = (a.n_out % 8 == 0 && reinterpret_cast<uintptr_t>(a.out) % 16 == 0 &&
                    (a.batch == 1 || ((size_t)a.out_stride * es) % 16 == 0)) ? 1 : 0;
    p.n_tiles = (a.N + 64 * H - 1) / (64 * H);
    p.items = (long long)a.m_vec * a.batch * p.n_tiles;
    return p;
}
// the work counter, and CTAs (clusters only where items are few)
bool too_many(long long items, int sms) {
    if (items + (long long)sms * kResident * kWarps <= 0x7fffffffLL) return false;
    set_error("problem too large for 32-bit tile ids");
    return true;
}
}  // namespace rows

// One wave of warps with few steps each: the copy is what counts.  Five steps per warp (2048 x 2048 half full, N = 49: 16.0 and 14.4 us; 1024 x 1024,
// N = 100: 10.3 and 12.3, in a graph 8.3 and 7.3) are as good as even, ten (512 x 4608 at 43 %) 13.9 and 14.4, in a graph 11.1 and 9.0.
// One or two columns are copied all the same: every warp asks for the same few lines (123 rows of 510 of 627, V = 16, N = 1 in a graph 11.7 us, copied 6.2;
// N = 3 6.9 and 6.3, from a stream 8.2 and 11.5).
constexpr long long kUnalignedSteps = 4;
bool sspmm_rows_reads_unaligned(const SpmmArgs& a, long long nvec) {
    const int sms = current_device_sm_count();
    if (sms <= 0 || nvec <= 0 || a.batch != 1 || a.m_vec <= 0 || a.n_out < 3 || reinterpret_cast<uintptr_t>(a.rhs) % 16 ||
        (int64_t)a.K * a.N * 2 > INT_MAX) return false;
    const rows::Route r = rows::route(a, nvec, sms);
    const long long steps = (nvec / a.m_vec + rows::kStep) / rows::kStep, warps = (long long)r.d.team * r.d.cluster;
    return r.way == rows::Route::kPlain && r.d.H == 1 && steps <= kUnalignedSteps * warps &&
           rows::count_items(&a, 1, 1) * warps <= (long long)sms * rows::kResident * rows::kWarps;
}
cudaError_t launch_sspmm_rows_unaligned(const SpmmArgs& a, long long nvec) {
    const int sms = current_device_sm_count();
    if (sms <= 0) return cudaErrorNoDevice;
    const rows::Division d = rows::route(a, nvec, sms).d;
    const rows::Problem p = rows::problem_of(a, 1);
    auto go = [&](auto v, auto out) {
        using OutT = decltype(out);
        constexpr int V = decltype(v)::value;
        static DeviceOnce once;
        return rows::launch_items<V, OutT, 1, rows::Tile<V, 1, sizeof(OutT) == 4>::kRawWarpBytes>(rows::sspmm_rows_unaligned_kernel<V, OutT>, once, p.items,
                                                                                                 d, a.stream, p, static_cast<OutT*>(a.out));
    };
    constexpr std::integral_constant<int, 8> k8{};
    constexpr std::integral_constant<int, 16> k16{};
    if (a.V == 16) return a.out_f16 ? go(k16, __half()) : go(k16, float());
    return a.out_f16 ? go(k8, __half()) : go(k8, float());
}

bool sspmm_rows_may_be_long(const SpmmArgs& a, long long nvec) {
    const int sms = current_device_sm_count() > 0 ? current_device_sm_count() : 148;
    return a.m_vec > 0 && rows::route(a, nvec, sms).long_rows;
}

// scratch: null, or sspmm_rows_scratch_bytes() bytes (long rows are then cut); nvec < 0: unknown.
cudaError_t launch_sspmm_rows(const SpmmArgs& a, long long nvec, void* scratch, bool spread) {
    const int sms = current_device_sm_count();
    if (sms <= 0) return cudaErrorNoDevice;
    const bool split = scratch != nullptr;
    rows::Route r = rows::route(a, nvec, sms);
    if (!spread) r.d = rows::divide(&a, 1, nvec, sms);
    if (split) r.way = rows::Route::kCut;
    else if (!spread || r.way == rows::Route::kCut) r.way = rows::Route::kPlain;
    const int H = split ? (a.N > 64 ? 2 : 1) : r.d.H;
    rows::Problem p = rows::problem_of(a, H);
    if (rows::too_many(p.items, sms)) return cudaErrorInvalidValue;
    if (split) {
        const rows::Scratch r = rows::plan_scratch(a, nvec);
        uint8_t* s = static_cast<uint8_t*>(scratch);
        p.chunk = r.chunk; p.cap_cut = r.cap_cut; p.cap_whole = r.cap_whole;
        p.header = reinterpret_cast<int*>(s);
        p.arrivals = reinterpret_cast<int*>(s + 16);
        p.entries = reinterpret_cast<int4*>(s + r.entries_at);
        p.partial = reinterpret_cast<float*>(s + r.partial_at);
    }
    if (a.V == 16)
        return a.out_f16 ? rows::launch_typed<16, __half>(a, p, H, r, sms) : rows::launch_typed<16, float>(a, p, H, r, sms);
    return a.out_f16 ? rows::launch_typed<8, __half>(a, p, H, r, sms) : rows::launch_typed<8, float>(a, p, H, r, sms);
}

RowsShape sspmm_rows_set_shape(const SpmmArgs* a, int count, long long nvec) {
    const rows::Division d = rows::divide(a, count, nvec, current_device_sm_count() > 0 ? current_device_sm_count() : 148);
    RowsShape r;
    r.columns = 64 * d.H; r.warps = d.team * d.cluster;
    r.items = rows::count_items(a, count, d.H);
    r.ctas = (r.items * d.team + rows::kWarps - 1) / rows::kWarps * d.cluster;
    return r;
}

cudaError_t launch_sspmm_rows_set(const SpmmArgs* a, int count, long long nvec) {
    const int sms = current_device_sm_count();
    if (sms <= 0) return cudaErrorNoDevice;
    const rows::Division d = rows::divide(a, count, nvec, sms);
    if (count > kRowsMaxSet || rows::too_many(rows::count_items(a, count, d.H), sms)) return cudaErrorInvalidValue;
    rows::ProblemSet s;
    s.count = count;
    s.first[0] = 0;
    for (int k = 0; k < count; ++k) {
        s.p[k] = rows::problem_of(a[k], d.H);
        s.out[k] = a[k].out;
        s.add[k] = a[k].add;
        s.first[k + 1] = s.first[k] + (int)s.p[k].items;
    }
    bool add = false;
    for (int k = 0; k < count; ++k) add = add || a[k].add;
    if (add) {
        if (!a->out_f16) { set_error("sums are added to fp16 results only"); return cudaErrorInvalidValue; }
        return a->V == 16 ? rows::launch_set<16, __half, true>(s, d, a->stream) : rows::launch_set<8, __half, true>(s, d, a->stream);
    }
    if (a->V == 16) return a->out_f16 ? rows::launch_set<16, __half, false>(s, d, a->stream) : rows::launch_set<16, float, false>(s, d, a->stream);
    return a->out_f16 ? rows::launch_set<8, __half, false>(s, d, a->stream) : rows::launch_set<8, float, false>(s, d, a->stream);
}

// ---- dense operands whose rows do not start on 16-byte boundaries -------------------------------
cudaError_t launch_align_rows(const SpmmArgs& a, int ld, __half* dst) {
    const int sms = current_device_sm_count();
    if (sms <= 0) return cudaErrorNoDevice;
    const int64_t blocks = ((int64_t)a.K * a.batch * (ld / 8) + 255) / 256;
    rows::align_rows_kernel<<<(unsigned)std::min<int64_t>(blocks, (int64_t)sms * 32), 256, 0, a.stream>>>(a.rhs, dst, a.K, a.N, ld, a.batch, a.rhs_stride);
    return cudaGetLastError();
}

}  // namespace sspmm_b200
