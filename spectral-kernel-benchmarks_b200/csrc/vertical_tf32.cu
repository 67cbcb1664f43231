// Split-TF32x3 grouped vertical GEMM for many small groups, on mma.sync.
//
// The tcgen05 form (tc_gemm.cu) is one pipeline per SM whose steps (unit tables,
// column cells, group image, 64-column tiles, epilogue) cost about 1.1 us per tile
// and 32 steps of the inner dimension however few columns a group has; it reaches
// its rate once a group has several hundred columns.  Here
// a tile is 32 complex columns of one group, several independent CTAs share an
// SM, and the group matrix is copied as plain FP32 (a quarter of the split,
// padded operand image's bytes) and split in registers.  mma.m16n8k8 TF32 runs at
// 277 TFLOP/s here, a quarter of tcgen05's rate, which is why large groups stay
// there (VerticalPlan chooses).  Measured, before (tcgen05) and now:
// vertical transforms both ways at 256^2, Nz 100, 173 -> 123 us (35 us of memory
// traffic); forward of 3 fields at 128^2, Nz 33, 20.5 -> 12.3 us.  A profile shows the
// issue slots 73 % busy: splitting and adding take several times the slots of the
// MMAs, so column tiles of 32 that share no split are what the next gain would need.
//
// Layout and roles are those of the FP64 form (vertical_f64.cu): D[r][n] =
// sum_s A[r][s] X[s][n] with a column's real and imaginary parts as neighbouring n,
// so a lane's result pairs are complex values; 8 warps, each two column tiles (8
// complex columns) and one half of the 16-row tiles; chunks of 32 inner steps in two
// cp.async stages.  Rows of 36 (or 8 j + 4) values make the A fragment loads (8
// rows x 4 steps) and the column fragment loads free of bank conflicts.  Matrices
// stored split, as (hi, lo) pairs, cost more in copies than the splitting (vertical
// GEMM at 256^2, Nz 100: 138 us against 128).
//
// Split precision as in tc_gemm.cu: x = hi + lo with hi = rna_tf32(x), lo =
// rna_tf32(x - hi), D = Ahi*Blo + Alo*Bhi + Ahi*Bhi.  Every 8 steps start from a
// zero accumulator and are added in FP32 registers (the tcgen05 form adds once per
// 32), so the accumulator's rounding enters over 8 products only.

#include <cstdint>

#include "launch.cuh"
#include "vertical_device.cuh"

namespace skb {
namespace {

constexpr int kTileCols = 32;
constexpr int kChunk = kGemmTf32Chunk;
constexpr int kPitch = kChunk + 4;
constexpr int kThreads = 256;

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
// One complex value, zeros where !ok.
__device__ __forceinline__ void copy_or_zero(void* dst, const void* src, bool ok) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
__device__ __forceinline__ uint32_t tf32_rna(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32_rna(x);
    lo = tf32_rna(x - __uint_as_float(hi));
}
// D = A B, and D += A B.
__device__ __forceinline__ void mma_first(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, "
        "%10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
        "%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int MH>
constexpr size_t stage_bytes() {
    return sizeof(float) * (size_t(2) * MH * 16 * kPitch + size_t(2) * kTileCols * kPitch);
}
template <int MH>
constexpr int resident() {
    const int regs = 65536 / (kThreads * (8 * MH + 40));
    const int smem = int(size_t(227 * 1024) / (2 * stage_bytes<MH>() + 2048));
    return regs < smem ? regs : smem;
}

// One chunk: kc steps of s (a multiple of 8) for MH row tiles (FULL: all of them
// exist, else `rows` do) and one or two column tiles.
template <int MH, bool FULL, bool TWO>
__device__ __forceinline__ void multiply(float (&acc)[MH][2][4], const float* a, const float* x, int kc, int row,
                                         int rows) {
#pragma unroll 1
    for (int s = 0; s < kc; s += 8, a += 8, x += 16) {
        uint32_t bh[2][2], bl[2][2];
#pragma unroll
        for (int n = 0; n < (TWO ? 2 : 1); ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) split(x[8 * h + n * 8 * kPitch], bh[n][h], bl[n][h]);
#pragma unroll
        for (int i = 0; i < MH; ++i) {
            if (FULL || i < rows) {
                const float* ai = a + 16 * i * row;
                uint32_t ah[4], al[4];
                split(ai[0], ah[0], al[0]);
                split(ai[8 * row], ah[1], al[1]);
                split(ai[4], ah[2], al[2]);
                split(ai[8 * row + 4], ah[3], al[3]);
#pragma unroll
                for (int n = 0; n < (TWO ? 2 : 1); ++n) {
                    float d[4];
                    mma_first(d, ah, bl[n]);
                    mma(d, al, bh[n]);
                    mma(d, ah, bh[n]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i][n][e] += d[e];
                }
            }
        }
    }
}

// Row tiles [0, MH) of 16 rows belong to warps 0-3, [MH, 2 MH) to warps 4-7.
template <int MH>
__global__ void __launch_bounds__(kThreads, resident<MH>())
    grouped_gemm_tf32_kernel(int R, int S, const float* __restrict__ images, GroupTiles tiles,
                             const float2* __restrict__ in, float2* __restrict__ out, BinBoundary inBins,
                             BinBoundary outBins) {
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
    const float* image = images + g * tiles.matrixStride;
    const int chunks = (S + kChunk - 1) / kChunk;
    auto stageA = [&](int b) { return reinterpret_cast<float*>(smem_raw + b * stage_bytes<MH>()); };
    auto stageX = [&](int b) { return stageA(b) + 2 * MH * 16 * kPitch; };

    auto issue = [&](int c, int b) {
        const int left = S - c * kChunk;
        const int steps = min(kChunk, (left + 7) & ~7);
        const float* src = image + static_cast<long long>(c) * kPitch * R;
        float* sA = stageA(b);
        for (int i = tid; i < R * (steps + 4) / 4; i += kThreads) copy16(sA + 4 * i, src + 4 * i);
        // Warp w copies columns w + 8 k, a lane one step of the chunk.
        if (lane < steps) {
            float* sX = stageX(b) + 2 * (warp * kPitch + lane);
            const float2* from = in + c * kChunk + lane;
            for (int col = warp; col < ncols; col += kThreads / 32, sX += 2 * kPitch * (kThreads / 32))
                copy_or_zero(sX, lane < left ? from + colIn[col] : in, lane < left);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // Warps w and w + 4 share a scheduler: their column pairs lie two apart, and
    // the pairs turn with the tile, so that part-filled tiles load the four
    // schedulers alike.
    const int np = (warp + 2 * (warp >> 2) + tile) & 3;  // columns 8 np .. 8 np + 7
    const int m0 = (warp >> 2) * MH;                     // first row tile
    const int mts = (R + 15) / 16 - m0;                  // row tiles that exist from there on
    const bool two = ncols > 8 * np + 4;                 // second column tile in use
    const bool any = ncols > 8 * np && mts > 0;
    float acc[MH][2][4];
#pragma unroll
    for (int i = 0; i < MH; ++i)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][n][e] = 0.f;

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
            // Fragment addresses: rows 16 (m0 + i) + lane/4 (+ 8), steps lane % 4
            // (+ 4); column 8 np + 4 n + lane/8, part (lane/4) % 2.
            const int kc = min(kChunk, (S - c * kChunk + 7) & ~7), row = kc + 4;
            const float* a = stageA(c & 1) + (16 * m0 + (lane >> 2)) * row + (lane & 3);
            const float* x = stageX(c & 1) + (8 * np + (lane >> 3)) * 2 * kPitch + 2 * (lane & 3) + ((lane >> 2) & 1);
            if (mts < MH) {
                two ? multiply<MH, false, true>(acc, a, x, kc, row, mts)
                    : multiply<MH, false, false>(acc, a, x, kc, row, mts);
            } else {
                two ? multiply<MH, true, true>(acc, a, x, kc, row, MH)
                    : multiply<MH, true, false>(acc, a, x, kc, row, MH);
            }
        }
        __syncthreads();
    }
    if (!any) return;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const int c = 8 * np + 4 * n + (lane & 3);
        if (c >= ncols) continue;
        float2* to = out + colOut[c];
        float2* partner = colPartner[c] >= 0 ? out + colPartner[c] : nullptr;
        const float sg = colConj[c] ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < MH; ++i) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 16 * (m0 + i) + 8 * h + (lane >> 2);
                if (r < R) {
                    const float re = acc[i][n][2 * h], im = sg * acc[i][n][2 * h + 1];
                    to[r] = make_float2(re, im);
                    if (partner != nullptr) partner[r] = make_float2(re, -im);
                }
            }
        }
    }
}

template <int MH>
cudaError_t launch_mh(int R, int S, const float* images, const GroupTiles& tiles, const float2* in, float2* out,
                      const BinBoundary& ib, const BinBoundary& ob, cudaStream_t stream) {
    auto kernel = grouped_gemm_tf32_kernel<MH>;
    const size_t bytes = 2 * stage_bytes<MH>();
    if (bytes > 48 * 1024) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
        if (err != cudaSuccess) return err;
    }
    return launch_chained(kernel, dim3(unsigned(tiles.tiles)), kThreads, bytes, stream, R, S, images, tiles, in, out, ib,
                          ob);
}

// natural [groups][R][S] -> images, one thread per (group, row, s of the padded row).
__global__ void tf32_image_kernel(const float* __restrict__ natural, long long groups, int R, int S, int row,
                                  float* __restrict__ images) {
    const long long total = groups * R * row;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long g = i / (static_cast<long long>(R) * row);
        const int at = static_cast<int>(i - g * R * row);
        const int chunk = at / (R * kPitch);
        const int left = S - chunk * kChunk;
        const int pitch = gemm_tf32_chunk_row(left);
        const int within = at - chunk * R * kPitch;
        const int r = within / pitch, s = within - r * pitch;
        images[i] = s < kChunk && s < left ? natural[(g * R + r) * S + chunk * kChunk + s] : 0.f;
    }
}

}  // namespace

cudaError_t gemm_tf32_build_images(const float* natural, long long groups, int R, int S, float* images,
                                   cudaStream_t stream) {
    if (groups <= 0) return cudaSuccess;
    const int row = gemm_tf32_row(S);
    const long long blocks = (groups * R * row + 255) / 256;
    tf32_image_kernel<<<unsigned(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, stream>>>(natural, groups, R, S, row,
                                                                                          images);
    return cudaGetLastError();
}

cudaError_t launch_grouped_gemm_tf32(int R, int S, const float* images, const GroupTiles& tiles, const float2* in,
                                     float2* out, const BinBoundary& ib, const BinBoundary& ob,
                                     cudaStream_t stream) {
    if (tiles.tiles <= 0) return cudaSuccess;
    switch (((R + 15) / 16 + 1) / 2) {
        case 1: return launch_mh<1>(R, S, images, tiles, in, out, ib, ob, stream);
        case 2: return launch_mh<2>(R, S, images, tiles, in, out, ib, ob, stream);
        case 3: return launch_mh<3>(R, S, images, tiles, in, out, ib, ob, stream);
        case 4: return launch_mh<4>(R, S, images, tiles, in, out, ib, ob, stream);
        case 5: return launch_mh<5>(R, S, images, tiles, in, out, ib, ob, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace skb
