// FP64 grouped vertical GEMM on the FP64 matrix instructions.  See vertical.hpp.
//
// One CTA of 8 warps computes a tile of up to 32 complex columns of one K^2
// group, all R output rows, as D[r][n] = sum_s A[r][s] X[s][n] with the real and
// imaginary parts of a column as neighbouring n: mma.m8n8k4 fragments then need
// no padding beyond 8 rows, 4 complex columns and 4 steps of s, and a lane's two
// results are one complex value.  Warp w takes two column tiles (8 complex
// columns) and one half of the row tiles.
//
// The inner dimension is streamed in chunks of kGemmF64Chunk = 28 through two
// shared-memory stages (cp.async).  The group matrices are stored chunk by chunk
// ([chunk][r][s of the chunk]), so a chunk is one contiguous run of 16-byte
// copies.  A row of 28 (or any odd multiple of 4) values makes the fragment loads
// (4 rows x 4 steps per access phase) free of bank conflicts, and a column of 28
// complex values those of the columns.
//
// Bound: latency and the barriers between chunks (at 16-32 warps per SM), then
// the FP64 pipe.  tcgen05 has no FP64 form; mma.m8n8k4 runs at 37.0 TFLOP/s here
// (FMA instructions 34.1) and a warp's 18 of them per step of 4 take 11 shared
// loads.  The FMA form before it padded rows to 32 and was held at 39-46 % of
// the FP64 pipe by shared loads and 8-byte copies.  Both directions at 256^2,
// Nz 65, 3 fields (2,045 groups of 17 columns): 156 -> 64 us; 512^2, Nz 129:
// 15-field inverse 2.14 -> 1.27 ms, 4-field forward 0.82 -> 0.37 ms.  Persistent
// CTAs with the copies running across tiles: 77 us (against 74 before a warp copied
// whole columns), and 1 % slower at 512^2.

#include "launch.cuh"
#include "vertical_device.cuh"

namespace skb {
namespace {

constexpr int kTileCols = 32;
constexpr int kChunk = kGemmF64Chunk;
constexpr int kThreads = 256;

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
// 8 or 16 bytes; zeros where !ok.
template <int BYTES>
__device__ __forceinline__ void copy_or_zero(void* dst, const void* src, bool ok) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    const int n = ok ? BYTES : 0;
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void mma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

template <int MH>
constexpr size_t stage_bytes() {
    return sizeof(double) * (size_t(2) * MH * 8 * kChunk + size_t(2) * kTileCols * kChunk);
}
// Resident CTAs: two accumulator tiles of 4 registers per row tile and thread.
template <int MH>
constexpr int resident() {
    const int regs = 65536 / (kThreads * (8 * MH + 40));
    const int smem = int(size_t(227 * 1024) / (2 * stage_bytes<MH>() + 2048));
    return regs < smem ? (regs < 1 ? 1 : regs) : smem;
}

// One chunk: kc steps of s for MH row tiles (FULL: all of them exist, else
// `rows` do) and one or two column tiles.
template <int MH, int KC, bool FULL, bool TWO>
__device__ __forceinline__ void multiply(double (&acc)[MH][2][2], const double* a, const double* x, int width,
                                         int pitch, int rows) {
    const int kc = KC > 0 ? KC : width, row = KC > 0 ? KC : pitch;
#pragma unroll(KC > 0 ? KC / 4 : 1)
    for (int s = 0; s < kc; s += 4) {
        const double x0 = x[2 * s];
        const double x1 = TWO ? x[2 * s + 8 * kChunk] : 0.0;
#pragma unroll
        for (int i = 0; i < MH; ++i) {
            if (FULL || i < rows) {
                const double av = a[8 * i * row + s];
                mma(acc[i][0], av, x0);
                if (TWO) mma(acc[i][1], av, x1);
            }
        }
    }
}

// Row tiles [0, MH) of 8 rows belong to warps 0-3, [MH, 2 MH) to warps 4-7.
template <int MH>
__global__ void __launch_bounds__(kThreads, resident<MH>())
    grouped_gemm_f64_kernel(int R, int S, const double* __restrict__ images, GroupTiles tiles, ComplexOperand in,
                            ComplexOperand out, BinBoundary inBins, BinBoundary outBins) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // Element offsets of each tile column's input and output (and the output
    // partner, or -1), and whether the output is conjugated.
    __shared__ long long colIn[kTileCols], colOut[kTileCols], colPartner[kTileCols];
    __shared__ bool colConj[kTileCols];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x;
    const int g = __ldg(tiles.tileGroup + tile);
    const int c0 = __ldg(tiles.tileColumn + tile);
    const int ncols = __ldg(tiles.tileCount + tile);
    if (tid < ncols) {
        long long col = c0 + tid;
        if (tiles.virtualColumns) {
            const int per = __ldg(tiles.tilePer + tile);
            const int member = (c0 + tid) / per;
            col = member * tiles.memberColumns + __ldg(tiles.tileFirst + tile) + (c0 + tid - member * per);
        }
        long long base = col * S, partner = -1;
        bool conjIn = false, conjOut = false;
        if (inBins.cell != nullptr) bin_column(inBins, static_cast<int>(col), base, partner, conjIn);
        colIn[tid] = base;
        base = col * R;
        partner = -1;
        if (outBins.cell != nullptr) bin_column(outBins, static_cast<int>(col), base, partner, conjOut);
        colOut[tid] = base;
        colPartner[tid] = partner;
        // The matrices are real: a conjugated input gives the conjugate product.
        colConj[tid] = conjIn != conjOut;
    }
    __syncthreads();
    const bool split = in.im != nullptr;
    const double* image = images + g * tiles.matrixStride;
    const int chunks = (S + kChunk - 1) / kChunk;
    auto stageA = [&](int b) { return reinterpret_cast<double*>(smem_raw + b * stage_bytes<MH>()); };
    auto stageX = [&](int b) { return stageA(b) + 2 * MH * 8 * kChunk; };

    auto issue = [&](int c, int b) {
        const int left = S - c * kChunk;
        const int steps = min(kChunk, (left + 3) & ~3);
        const double* src = image + static_cast<long long>(c) * kChunk * R;
        double* sA = stageA(b);
        for (int i = tid; i < R * gemm_f64_chunk_row(left) / 2; i += kThreads) copy16(sA + 2 * i, src + 2 * i);
        // Warp w copies columns w + 8 k, a lane one step of the chunk.
        if (lane < steps) {
            const bool ok = lane < left;
            const int first = c * kChunk + lane;
            double* sX = stageX(b) + 2 * (warp * kChunk + lane);
            for (int col = warp; col < ncols; col += kThreads / 32, sX += 2 * kChunk * (kThreads / 32)) {
                const long long at = ok ? colIn[col] + first : 0;
                if (split) {
                    copy_or_zero<8>(sX, static_cast<const double*>(in.re) + at, ok);
                    copy_or_zero<8>(sX + 1, static_cast<const double*>(in.im) + at, ok);
                } else {
                    copy_or_zero<16>(sX, static_cast<const double2*>(in.re) + at, ok);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // Warps w and w + 4 share a scheduler: their column pairs lie two apart, and
    // the pairs turn with the tile, so that part-filled tiles load the four
    // schedulers alike.
    const int np = (warp + 2 * (warp >> 2) + tile) & 3;  // columns 8 np .. 8 np + 7
    const int m0 = (warp >> 2) * MH;                     // first row tile
    const int mts = (R + 7) / 8 - m0;                    // row tiles that exist from there on
    const bool two = ncols > 8 * np + 4;                 // second column tile in use
    const bool any = ncols > 8 * np && mts > 0;
    double acc[MH][2][2];
#pragma unroll
    for (int i = 0; i < MH; ++i)
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[i][n][0] = acc[i][n][1] = 0.0;

    grid_wait();
    issue(0, 0);
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            issue(c + 1, (c + 1) & 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (any) {
            // Fragment addresses: row 8 (m0 + i) + lane/4, step lane % 4; column
            // 8 np + 4 n + lane/8, part (lane/4) % 2.
            const int left = S - c * kChunk;
            const int kc = min(kChunk, (left + 3) & ~3), row = gemm_f64_chunk_row(left);
            const double* a = stageA(c & 1) + (8 * m0 + (lane >> 2)) * row + (lane & 3);
            const double* x = stageX(c & 1) + (8 * np + (lane >> 3)) * 2 * kChunk + 2 * (lane & 3) + ((lane >> 2) & 1);
            if (mts < MH) {
                two ? multiply<MH, 0, false, true>(acc, a, x, kc, row, mts)
                    : multiply<MH, 0, false, false>(acc, a, x, kc, row, mts);
            } else if (kc == kChunk) {
                two ? multiply<MH, kChunk, true, true>(acc, a, x, kc, row, MH)
                    : multiply<MH, kChunk, true, false>(acc, a, x, kc, row, MH);
            } else {
                two ? multiply<MH, 0, true, true>(acc, a, x, kc, row, MH)
                    : multiply<MH, 0, true, false>(acc, a, x, kc, row, MH);
            }
        }
        __syncthreads();
    }
    if (!any) return;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const int c = 8 * np + 4 * n + (lane & 3);
        if (c >= ncols) continue;
        const long long to = colOut[c], partner = colPartner[c];
        const bool conj = colConj[c];
#pragma unroll
        for (int i = 0; i < MH; ++i) {
            const int r = 8 * (m0 + i) + (lane >> 2);
            if (r < R) {
                const double re = acc[i][n][0], im = conj ? -acc[i][n][1] : acc[i][n][1];
                if (split) {
                    static_cast<double*>(out.re)[to + r] = re;
                    static_cast<double*>(out.im)[to + r] = im;
                    if (partner >= 0) {
                        static_cast<double*>(out.re)[partner + r] = re;
                        static_cast<double*>(out.im)[partner + r] = -im;
                    }
                } else {
                    static_cast<double2*>(out.re)[to + r] = make_double2(re, im);
                    if (partner >= 0) static_cast<double2*>(out.re)[partner + r] = make_double2(re, -im);
                }
            }
        }
    }
}

template <int MH>
cudaError_t launch_mh(int R, int S, const double* images, const GroupTiles& tiles, ComplexOperand in,
                      ComplexOperand out, const BinBoundary& ib, const BinBoundary& ob, cudaStream_t stream) {
    auto kernel = grouped_gemm_f64_kernel<MH>;
    const size_t bytes = 2 * stage_bytes<MH>();
    if (bytes > 48 * 1024) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
        if (err != cudaSuccess) return err;
    }
    return launch_chained(kernel, dim3(unsigned(tiles.tiles)), kThreads, bytes, stream, R, S, images, tiles, in, out, ib,
                          ob);
}

}  // namespace

cudaError_t launch_grouped_gemm_f64(int R, int S, const double* images, const GroupTiles& tiles, ComplexOperand in,
                                    ComplexOperand out, const BinBoundary& ib, const BinBoundary& ob,
                                    cudaStream_t stream) {
    if ((in.im != nullptr) != (out.im != nullptr)) return cudaErrorInvalidValue;
    switch (((R + 7) / 8 + 1) / 2) {
        case 1: return launch_mh<1>(R, S, images, tiles, in, out, ib, ob, stream);
        case 2: return launch_mh<2>(R, S, images, tiles, in, out, ib, ob, stream);
        case 3: return launch_mh<3>(R, S, images, tiles, in, out, ib, ob, stream);
        case 4: return launch_mh<4>(R, S, images, tiles, in, out, ib, ob, stream);
        case 5: return launch_mh<5>(R, S, images, tiles, in, out, ib, ob, stream);
        case 6: return launch_mh<6>(R, S, images, tiles, in, out, ib, ob, stream);
        case 7: return launch_mh<7>(R, S, images, tiles, in, out, ib, ob, stream);
        case 8: return launch_mh<8>(R, S, images, tiles, in, out, ib, ob, stream);
        case 9: return launch_mh<9>(R, S, images, tiles, in, out, ib, ob, stream);
        case 10:
        case 11:
        case 12:
        case 13: return launch_mh<13>(R, S, images, tiles, in, out, ib, ob, stream);
        case 14:
        case 15:
        case 16:
        case 17:
        case 18: return launch_mh<18>(R, S, images, tiles, in, out, ib, ob, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace skb
