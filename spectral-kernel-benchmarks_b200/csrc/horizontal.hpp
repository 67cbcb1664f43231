// Launch interface of the horizontal (x/y) transform kernels.
//
// Two kernels make every horizontal operator:
//   row kernels     length-Nx r2c / c2r along x for B planes at one y,
//                   reading/writing real planes [plane][y][x] and a dense bin
//                   array [y][kx][plane] that keeps kx < K.
//   column kernels  length-Ny c2c along y for B planes of one kx column,
//                   reading either a dense bin array or retained modes
//                   (zero-fill + kx = 0 Hermitian repair), and writing either a
//                   dense bin array or retained modes (conjugation + scale).
// With K = Nx/2+1 and the dense array laid out as the WVM spectrum this is the
// full 2-D r2c/c2r (fftw_provider.cpp:537-610); with K = the active kx band and
// retained-mode I/O it is the pruned transform (pruned_fftw_provider.cpp:315-517).

#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace skb {

constexpr int kMaxViews = 128;

// One field of retained (compact) coefficients: element (mode, z) lives at
// z + modeStride*mode.  Interleaved complex when imag == nullptr (re points at
// the complex array), split real/imaginary arrays otherwise.
struct FieldView {
    void* re;
    void* im;
    long long modeStride;
};

struct ViewSet {
    FieldView v[kMaxViews];
    int count;
};

struct ModeTables {
    // cell map for embedding: map[kx*Ny + ky] = (mode << 1 | conj), or -1.
    const int* cellMap;
    // per-kx gather lists: entries colStart[kx] .. colStart[kx+1]-1 of
    // colKy[] and colMode[] (mode << 1 | conj).
    const int* colStart;
    const int* colKy;
    const int* colMode;
    // gather map: map[kx*Ny + ky] = (mode << 1 | conj) for stored cells only, or -1.
    const int* gatherMap;
};

enum class Precision { f64 = 0, f32 = 1 };

struct DenseBins {
    void* data;          // complex T
    long long planes;    // stride between consecutive kx (total planes, or planes of a block)
    long long kxStride;  // number of kx entries per ky row
    // Plane-blocked arrays (the plans' scratch): blocks of 2^blockShift planes,
    // each a [ky][kx][plane of the block] array of blockStride elements.
    int blockShift = 0;
    long long blockStride = 0;  // 0: one array, all planes innermost
    __host__ __device__ long long offset(long long plane) const {
        if (blockStride == 0) return plane;
        const long long block = plane >> blockShift;
        return block * blockStride + (plane - (block << blockShift));
    }
};

// Elements of a length-n sequence that one thread of the register-ended FFT
// holds (fft_regs.cuh).  Lengths up to 16 stay in one thread; 16 elements make
// 128- and 256-point transforms one exchange.  FP64 512-point columns hold 8:
// 16 would need twice the registers for the same two exchanges.
constexpr int regs_per_thread(int n) { return n <= 16 ? n : n <= 64 ? 8 : 16; }
constexpr int column_regs_per_thread(int n, bool f64) { return n == 512 && f64 ? 8 : regs_per_thread(n); }
// Row kernels (half-length m = Nx/2): elements per thread and the radix of the
// pass that runs along the planes.
constexpr int row_regs_per_thread(int m) { return m <= 16 ? m : m == 32 ? 8 : 16; }
constexpr int row_plane_radix(int m) {
    return m <= 16 ? m : m <= 64 ? 4 : m == 128 ? 8 : m == 256 ? 16 : 2;
}
// Twiddle table of those kernels: entry i is exp(-2 pi i k / n) with
// k = regs_table_index(n, perThread, first, i).  Pass after pass, [r - 1][j]
// with r < R, j < Ns and k = j r n / (Ns R); Ns is the product of the radices
// before the pass.  The first radix is `first` (perThread when 0), the others
// are perThread or what remains.
constexpr int regs_table_size(int n, int perThread, int first = 0) {
    const int ns = first > 0 ? first : perThread;
    return n > ns ? n - ns : 1;
}
constexpr int regs_table_index(int n, int perThread, int first, int i) {
    for (int ns = first > 0 ? first : perThread; ns < n;) {
        const int radix = n / ns < perThread ? n / ns : perThread;
        if (i < ns * (radix - 1)) return (i % ns) * (i / ns + 1) * (n / (ns * radix));
        i -= ns * (radix - 1);
        ns *= radix;
    }
    return 0;
}
// Where the entries of the pass with sub-transform size ns begin (radices
// perThread, perThread, ... from the first).
constexpr int regs_table_offset(int perThread, int ns) { return ns - perThread; }

// x-direction transforms.  Planes [0, planes) of real volumes laid out
// [plane][y][x]; bins kept for kx < keep.  twHalf and the column transforms' tw
// are tables in regs_table_index order: (Nx/2, row_regs_per_thread) forward,
// the same with first radix row_plane_radix inverse, and (Ny,
// column_regs_per_thread); twFull is the natural Nx-point table.
cudaError_t launch_rows_forward(Precision p, int nx, int ny, long long planes, int keep, const void* real,
                                DenseBins bins, const void* twHalf, const void* twFull, cudaStream_t stream);
cudaError_t launch_rows_inverse(Precision p, int nx, int ny, long long planes, int keep, DenseBins bins, void* real,
                                const void* twHalf, const void* twFull, cudaStream_t stream);
// One target of the flux: `in` holds the bins of three derivative slots of
// every member (slot 3 m + f, nz planes each), `velocity` the real volumes of U, V and
// W in the same slot order; `out` gets the bins of -scale (u q_x + v q_y + w q_z), nz
// planes per member.
cudaError_t launch_rows_product(Precision p, int nx, int ny, int nz, int members, int keep, double scale,
                                const void* velocity, DenseBins in, DenseBins out, const void* twInverse,
                                const void* twForward, const void* twFull, cudaStream_t stream);

// y-direction transforms over kx in [0, columns).
// sign = -1 forward, +1 inverse.
cudaError_t launch_columns_dense(Precision p, int sign, int ny, int columns, long long planes, DenseBins in,
                                 DenseBins out, const void* tw, cudaStream_t stream);
// Inverse: retained views -> dense bins (zero fill + Hermitian repair).
cudaError_t launch_columns_embed(Precision p, int ny, int nz, int columns, const ViewSet& views,
                                 const ModeTables& tables, DenseBins out, const void* tw, cudaStream_t stream);
// Forward: dense bins -> retained views (conjugation, scale).
cudaError_t launch_columns_gather(Precision p, int ny, int nz, int columns, DenseBins in, const ViewSet& views,
                                  const ModeTables& tables, double scale, const void* tw, cudaStream_t stream);

// Retention / embedding directly on a dense WVM spectrum (no transform).
cudaError_t launch_gather_dense(Precision p, int ny, int nz, long long modes, const int* modeKx, const int* modeKy,
                                const unsigned char* modeConj, DenseBins in, const ViewSet& views, double scale,
                                cudaStream_t stream);
cudaError_t launch_embed_dense(Precision p, int ny, int nz, int columns, const ViewSet& views,
                               const ModeTables& tables, DenseBins out, cudaStream_t stream);

// Largest supported power-of-two transform length along x (Nx) and y (Ny).
constexpr int kMaxLength = 2048;
bool supported_length(long long n);

}  // namespace skb
