// Horizontal transform kernels (row r2c/c2r along x, column c2c along y with
// fused retention/embedding).  See horizontal.hpp for the decomposition and
// fft_regs.cuh for the register-ended FFT.

#include "horizontal.hpp"

#include "fft_regs.cuh"
#include "launch.cuh"

namespace skb {
namespace {

// Lanes of one shared-memory access phase (128 bytes of complex values): the
// plane batch of a CTA is a multiple of it, so that global accesses along the
// planes move whole 128-byte pieces.
template <typename T>
constexpr int phase_lanes() {
    return 128 / int(sizeof(cx<T>));
}

// Resident CTAs per SM that a kernel is compiled for: what
// shared memory, the registers it needs (per thread, by elements held) and the
// thread limit allow.  At these counts ptxas
// spills 32 bytes in the 256-point FP64 inverse rows, 8 and 24 in the 128-point FP32
// columns of the pruned transforms and 4 or 8 in five other FP64 kernels.
template <typename T>
constexpr int resident_ctas(int threads, size_t bytes, int elements) {
    const int regs = sizeof(T) == 8 ? (elements > 8 ? 96 : 64) : (elements > 8 ? 56 : 40);
    int ctas = int(size_t(227 * 1024) / (bytes + 1024));
    if (65536 / (threads * regs) < ctas) ctas = 65536 / (threads * regs);
    if (2048 / threads < ctas) ctas = 2048 / threads;
    return ctas < 1 ? 1 : ctas > 16 ? 16 : ctas;
}

// ---------------------------------------------------------------------------
// Row kernels: M = Nx/2 complex points per row, B planes of one y per CTA.
//
// A row side and a plane side share the FFT.  On the row side T = M / E threads
// (lanes of one warp) hold a row's elements t + T e, so that global accesses of
// real rows run along x; on the plane side B consecutive lanes hold one bin of
// B planes, so that global accesses of bins run along the planes.  The exchange
// before the last pass (forward) or after the first one (inverse) is also the
// turn from one side to the other: one shared-memory write and read per element
// where a separate transpose tile took two more.  The plane side's radix-R pass
// has Ns = M / R butterflies j over the bins j + Ns r; bin M - k of k = j + Ns r
// belongs to butterfly Ns - j, so the real-spectrum split pairs butterflies
// {j, Ns - j} in one thread's registers ({0, Ns/2} pair within themselves), or,
// where a thread holds one butterfly only (M = 256), in two lanes that swap the
// upper half of their values.
//
// Bound: latency, at 20 warps per SM (96 registers in FP64), then HBM.  FP64,
// 516 planes of 512^2 kept to 171 bins (1.76 GB per launch): forward 426 ->
// 301 us (5.9 TB/s), inverse 541 -> 354 us (5.0 TB/s) against the radix-8
// kernels with every pass in shared memory; 195 planes of 256^2, all 129 bins:
// 51 / 54 -> 37 / 39 us.  Persistent CTAs with the tables in shared memory and
// the next tile's loads issued early ran 420 / 391 us, plane chunks sized for
// L2 ran slower at every size (16 to 192 planes).
template <typename T, int M>
struct RowShape {
    using V = cx<T>;
    static constexpr int E = row_regs_per_thread(M);
    static constexpr int TPR = M / E;  // row-side threads per row, at most 32
    static constexpr int L = phase_lanes<T>();
    static constexpr int B = TPR == 1 ? 32 : (128 / TPR > L) ? 128 / TPR : L;
    static constexpr int NT = B * TPR;
    static_assert(TPR <= 32 && E % 2 == 0 && B % L == 0, "a row's lanes form (part of) one warp");
    static constexpr int R = row_plane_radix(M);
    static constexpr int Ns = M / R;
    static constexpr int NB = E / R;  // butterflies per plane-side thread
    static constexpr size_t kBytes = TPR > 1 ? size_t(M) * B * sizeof(V) : 0;
    static constexpr int kCtas = resident_ctas<T>(NT, kBytes, E);
    // Position i of plane b in the exchange.  The swizzle spreads both sides'
    // accesses over the banks: row lanes write positions E apart or walk
    // consecutive ones (L / TPR planes per access phase when rows are short).
    static constexpr int kMul = TPR < L ? L / TPR : 1;
    static __device__ __forceinline__ int slot(int i, int b) { return i * B + (b ^ (((i ^ (i / E)) * kMul) & (L - 1))); }
};

// A row's own exchange among its lanes (512-point halves need two exchanges).
template <typename S>
struct RowExchange {
    typename S::V* x;
    int b;
    __device__ __forceinline__ void store(int i, typename S::V v) { x[S::slot(i, b)] = v; }
    __device__ __forceinline__ typename S::V load(int i) const { return x[S::slot(i, b)]; }
    __device__ __forceinline__ void fence() const { __syncwarp(); }
};

// Butterfly of plane-side thread g when it holds one (M = 256): pairs
// {j, 16 - j} in neighbouring groups of B lanes, 0 and 8 last.
__device__ __forceinline__ int paired_butterfly(int g) {
    const int h = g / 2 + 1;
    return g >= 14 ? (g - 14) * 8 : (g & 1) ? 16 - h : h;
}

// Lane whose butterfly holds bin M - k (0 and 8: the lane itself).
template <int B>
__device__ __forceinline__ int pair_source(int j) {
    const int lane = threadIdx.x & 31;
    return (j & 7) == 0 ? lane : lane ^ B;
}

// Row forward: real rows of length NX = 2M -> bins kx in [0, keep).
// Grid (plane chunks, ny).  The real row is read as M complex pairs
// z[m] = x[2m] + i x[2m+1], transformed, then split into the real spectrum:
//   X[k] = s + W^k o,  X[M-k] = conj(s - W^k o),  W = e^{-2 pi i/NX},
//   s = (Z[k] + conj Z[M-k])/2,  o = -i (Z[k] - conj Z[M-k])/2.
//
// row_forward: v holds the row side's elements; out is bin 0 of the plane side's
// plane (bins `stride` apart), written where live.
template <typename T, int M>
__device__ __forceinline__ void row_forward(cx<T> (&v)[RowShape<T, M>::E], cx<T>* data, cx<T>* out, long long stride,
                                            bool live, int keep, const cx<T>* __restrict__ tw,
                                            const cx<T>* __restrict__ twFull) {
    using V = cx<T>;
    using S = RowShape<T, M>;
    constexpr int R = S::R, Ns = S::Ns;
    const int tid = threadIdx.x;
    if constexpr (S::TPR > 1) {
        RowExchange<S> xch{data, tid / S::TPR};
        fft_regs_head<T, M, S::E, -1, Ns>(v, tid % S::TPR, tw, xch);
        __syncthreads();
    }
    const int b = tid % S::B;
    const int g = tid / S::B;
    auto split = [&](int k, V zk, V zmk) {
        const V zm = cconj(zmk);
        const V s = cscale(cadd(zk, zm), T(0.5));
        const V d = csub(zk, zm);
        const V wo = cmul(__ldg(twFull + k), V{T(0.5) * d.y, T(-0.5) * d.x});
        if (live && k < keep) out[stride * k] = cadd(s, wo);
        if (live && 2 * k != M && M - k < keep) out[stride * (M - k)] = cconj(csub(s, wo));
    };
    auto split0 = [&](V z0) {
        if (live) out[0] = {z0.x + z0.y, T(0)};
        if (live && M < keep) out[stride * M] = {z0.x - z0.y, T(0)};
    };
    // Last pass of butterfly j: bins j + Ns r.
    auto last = [&](int j, V* u) {
#pragma unroll
        for (int r = 0; r < R; ++r) u[r] = data[S::slot(j + Ns * r, b)];
        const V* w = tw + regs_table_offset(S::E, Ns) + j;
#pragma unroll
        for (int r = 1; r < R; ++r) u[r] = cmul(u[r], twiddle<-1>(w, Ns * (r - 1)));
        dft_small<-1, R>(u);
    };
    if constexpr (S::TPR == 1) {
        dft_small<-1, M>(v);
        split0(v[0]);
#pragma unroll
        for (int k = 1; k <= M / 2; ++k) split(k, v[k], v[M - k]);
    } else if constexpr (S::NB == 1) {
        const int j = paired_butterfly(g);
        const int src = pair_source<S::B>(j);
        last(j, v);
        const V half = v[R / 2];
        if (j == 0) {
            // Bin M - k of k = Ns r is register R - r: one up, like the other lanes'.
#pragma unroll
            for (int e = R / 2; e < R - 1; ++e) v[e] = v[e + 1];
        }
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
            const V other = {__shfl_sync(0xFFFFFFFFu, v[R - 1 - r].x, src), __shfl_sync(0xFFFFFFFFu, v[R - 1 - r].y, src)};
            if (r > 0 || j > 0) split(j + Ns * r, v[r], other);
        }
        if (j == 0) {
            split0(v[0]);
            split(M / 2, half, half);
        }
    } else {
#pragma unroll
        for (int i = 0; i < S::NB / 2; ++i) {
            const int q = g + S::TPR * i;
            V a[R], c[R];
            last(q, a);
            last(q == 0 ? Ns / 2 : Ns - q, c);
            if (i == 0 && q == 0) {
                split0(a[0]);
#pragma unroll
                for (int r = 1; r <= R / 2; ++r) split(Ns * r, a[r], a[R - r]);
#pragma unroll
                for (int r = 0; r < R / 2; ++r) split(Ns / 2 + Ns * r, c[r], c[R - 1 - r]);
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) split(q + Ns * r, a[r], c[R - 1 - r]);
            }
        }
    }
}

// Row inverse: bins kx in [0, keep) (zero above) -> real rows, unnormalised,
// with FFTW's c2r semantics (imaginary parts of the kx = 0 and kx = NX/2 bins
// are ignored).  Pre-process Z[k] = s + i t, Z[M-k] = conj(s - i t) with
// s = X[k] + conj X[M-k], t = e^{+2 pi i k/NX} (X[k] - conj X[M-k]), then an
// inverse length-M FFT gives x[2m] + i x[2m+1].  The radices run in the
// forward kernel's order reversed, so the plane side has the same butterflies.
//
// row_inverse: in is bin 0 of the plane side's plane (bins `stride` apart), read
// where live; leaves the row side's elements in v.  `between` runs between the two
// sides (loads to have in flight during the row side's passes).
template <typename T, int M, typename F>
__device__ __forceinline__ void row_inverse(cx<T> (&v)[RowShape<T, M>::E], cx<T>* data, const cx<T>* in,
                                            long long stride, bool live, int keep, const cx<T>* __restrict__ tw,
                                            const cx<T>* __restrict__ twFull, F between) {
    using V = cx<T>;
    using S = RowShape<T, M>;
    constexpr int R = S::R, Ns = S::Ns;
    const int tid = threadIdx.x;
    {
        const int b = tid % S::B;
        const int g = tid / S::B;
        auto load = [&](int k) -> V { return live && k < keep ? in[stride * k] : V{T(0), T(0)}; };
        // (X[k], X[M-k]) -> (Z[k], Z[M-k])
        auto merge = [&](int k, V& xk, V& xm) {
            const V s = cadd(xk, cconj(xm));
            const V w = cmulc(csub(xk, cconj(xm)), __ldg(twFull + k));
            xk = {s.x - w.y, s.y + w.x};
            xm = {s.x + w.y, w.x - s.y};
        };
        // Bins 0 and NX/2 are real.
        auto merge0 = [&](V& x0, V xn) { x0 = {x0.x + xn.x, x0.x - xn.x}; };
        // First pass of butterfly j (positions j R + r of the exchange).
        auto first = [&](int j, V* u) {
            dft_small<+1, R>(u);
#pragma unroll
            for (int r = 0; r < R; ++r) data[S::slot(j * R + r, b)] = u[r];
        };
        if constexpr (S::TPR == 1) {
#pragma unroll
            for (int k = 0; k < M; ++k) v[k] = load(k);
            merge0(v[0], load(M));
#pragma unroll
            for (int k = 1; k <= M / 2; ++k) {
                V xm = v[M - k];
                merge(k, v[k], xm);
                if (2 * k != M) v[M - k] = xm;
            }
            dft_small<+1, M>(v);
        } else if constexpr (S::NB == 1) {
            const int j = paired_butterfly(g);
            const int src = pair_source<S::B>(j);
            // Butterfly 0 holds the partners one register up: its upper half is
            // loaded (and put back) shifted, bin NX/2 last, bin M/2 apart.
            V half = j == 0 ? load(M / 2) : V{T(0), T(0)};
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = load(j + Ns * r + (r >= R / 2 && j == 0 ? Ns : 0));
#pragma unroll
            for (int r = 0; r < R / 2; ++r) {
                V& up = v[R - 1 - r];
                V other = {__shfl_sync(0xFFFFFFFFu, up.x, src), __shfl_sync(0xFFFFFFFFu, up.y, src)};
                if (r == 0 && j == 0)
                    merge0(v[0], other);
                else
                    merge(j + Ns * r, v[r], other);
                // Z[M-k] goes back to the lane that X[M-k] came from.
                up = {__shfl_sync(0xFFFFFFFFu, other.x, src), __shfl_sync(0xFFFFFFFFu, other.y, src)};
            }
            if (j == 0) {
                V self = half;
                merge(M / 2, half, self);
#pragma unroll
                for (int e = R - 1; e > R / 2; --e) v[e] = v[e - 1];
                v[R / 2] = half;
            }
            first(j, v);
        } else {
#pragma unroll
            for (int i = 0; i < S::NB / 2; ++i) {
                const int q = g + S::TPR * i;
                const int qc = q == 0 ? Ns / 2 : Ns - q;
                V* a = v + 2 * R * i;
                V* c = a + R;
#pragma unroll
                for (int r = 0; r < R; ++r) a[r] = load(q + Ns * r);
#pragma unroll
                for (int r = 0; r < R; ++r) c[r] = load(qc + Ns * r);
            }
#pragma unroll
            for (int i = 0; i < S::NB / 2; ++i) {
                const int q = g + S::TPR * i;
                const int qc = q == 0 ? Ns / 2 : Ns - q;
                V* a = v + 2 * R * i;
                V* c = a + R;
                if (i == 0 && q == 0) {
                    merge0(a[0], load(M));
#pragma unroll
                    for (int r = 1; r < R / 2; ++r) merge(Ns * r, a[r], a[R - r]);
                    V self = a[R / 2];
                    merge(M / 2, a[R / 2], self);
#pragma unroll
                    for (int r = 0; r < R / 2; ++r) merge(Ns / 2 + Ns * r, c[r], c[R - 1 - r]);
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) merge(q + Ns * r, a[r], c[R - 1 - r]);
                }
                first(q, a);
                first(qc, c);
            }
        }
    }
    between();
    if constexpr (S::TPR > 1) {
        const int t = tid % S::TPR;
        __syncthreads();
        RowExchange<S> xch{data, tid / S::TPR};
#pragma unroll
        for (int e = 0; e < S::E; ++e) v[e] = xch.load(t + S::TPR * e);
        fft_regs<T, M, S::E, +1, R>(v, t, tw, xch);
    }
}

// Grid (plane chunks, ny).
template <typename T, int M>
__global__ void __launch_bounds__(RowShape<T, M>::NT, RowShape<T, M>::kCtas)
    rows_forward_kernel(int ny, long long planes, int keep, const T* __restrict__ real, DenseBins bins,
                        const cx<T>* __restrict__ tw, const cx<T>* __restrict__ twFull) {
    using V = cx<T>;
    using S = RowShape<T, M>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long p0 = (long long)blockIdx.x * S::B;
    const int y = blockIdx.y;
    V v[S::E];
    grid_wait();
    const long long row = p0 + threadIdx.x / S::TPR;
    if (row < planes) {
        const V* from = reinterpret_cast<const V*>(real + (row * ny + y) * (2 * M)) + threadIdx.x % S::TPR;
#pragma unroll
        for (int e = 0; e < S::E; ++e) v[e] = from[S::TPR * e];
    } else {
#pragma unroll
        for (int e = 0; e < S::E; ++e) v[e] = {T(0), T(0)};
    }
    const long long p = p0 + threadIdx.x % S::B;
    const bool live = p < planes;
    V* out = reinterpret_cast<V*>(bins.data) + bins.offset(live ? p : 0) + bins.planes * bins.kxStride * y;
    row_forward<T, M>(v, reinterpret_cast<V*>(smem_raw), out, bins.planes, live, keep, tw, twFull);
}

template <typename T, int M>
__global__ void __launch_bounds__(RowShape<T, M>::NT, RowShape<T, M>::kCtas)
    rows_inverse_kernel(int ny, long long planes, int keep, DenseBins bins, T* __restrict__ real,
                        const cx<T>* __restrict__ tw, const cx<T>* __restrict__ twFull) {
    using V = cx<T>;
    using S = RowShape<T, M>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long p0 = (long long)blockIdx.x * S::B;
    const int y = blockIdx.y;
    V v[S::E];
    grid_wait();
    const long long p = p0 + threadIdx.x % S::B;
    const bool live = p < planes;
    const V* in = reinterpret_cast<const V*>(bins.data) + bins.offset(live ? p : 0) + bins.planes * bins.kxStride * y;
    row_inverse<T, M>(v, reinterpret_cast<V*>(smem_raw), in, bins.planes, live, keep, tw, twFull, [] {});
    const long long row = p0 + threadIdx.x / S::TPR;
    if (row >= planes) return;
    V* to = reinterpret_cast<V*>(real + (row * ny + y) * (2 * M)) + threadIdx.x % S::TPR;
#pragma unroll
    for (int e = 0; e < S::E; ++e) to[S::TPR * e] = v[e];
}

// One target of the staged flux, for B planes (member m, level z) of one y: the rows
// of the three derivative slots are transformed one after the other and multiplied,
// in registers, by the rows of U, V and W; the negated, scaled sum goes back through
// the forward transform to the target's bins:
//   bins(m, z) <- r2c(-scale (u q_x + v q_y + w q_z)),  q_f = c2r(bins(3 m + f, z)).
// Neither the derivatives' real rows nor the product's are stored: 8 of the 11 real
// volumes that inverse rows, pointwise product and forward rows moved per target.
// Bound: latency, at two CTAs of 128 threads per SM (FP64, 255 registers and, at 512
// points, 100 bytes of spills: the sum, a slot's row and the velocity row in flight; FP32
// at 512 points 128 registers and 56 bytes), 3.6 TB/s.  Row stages of a flux, before
// and now: FP64 512^2, Nz 129, 4 targets 2869 -> 2005 us, 256^2, Nz 65, 3 targets of 2
// members 597 -> 390; FP32 512^2, Nz 65 842 -> 686, 256^2 337 -> 225; FP64 1024^2, Nz
// 17 1324 -> 1235, FP32 836 -> 877 (1141 with every pass of the rows in shared
// memory).  The row bodies shared with this kernel made the plain row kernels up to
// 2 % slower (FP32 256^2 pruned round trip 60.4 -> 61.7 us, FP64 256^2 FFT 166.5 -> 168).  512^2 without the L2 prefetches 2400, with 168 registers for a third CTA
// (spills) 2037-2051.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <typename T, int M>
struct ProductShape {
    using S = RowShape<T, M>;
    static constexpr int regs = sizeof(T) == 8 ? (S::E > 8 ? 255 : 128) : (S::E > 8 ? 128 : 80);
    static constexpr int bySmem = int(size_t(227 * 1024) / (S::kBytes + 1024));
    static constexpr int byRegs = 65536 / (S::NT * regs);
    static constexpr int least = bySmem < byRegs ? bySmem : byRegs;
    static constexpr int kCtas = least < 1 ? 1 : least > 16 ? 16 : least;
};

template <typename T, int M>
__global__ void __launch_bounds__(RowShape<T, M>::NT, ProductShape<T, M>::kCtas)
    rows_product_kernel(int ny, int nz, long long planes, int keep, T scale, const T* __restrict__ velocity,
                        DenseBins in, DenseBins bins, const cx<T>* __restrict__ twInverse,
                        const cx<T>* __restrict__ twForward, const cx<T>* __restrict__ twFull) {
    using V = cx<T>;
    using S = RowShape<T, M>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* data = reinterpret_cast<V*>(smem_raw);
    const long long p0 = (long long)blockIdx.x * S::B;
    const int y = blockIdx.y;
    // Plane side: this thread's target plane and slot 0's plane of it.
    const long long p = p0 + threadIdx.x % S::B;
    const bool live = p < planes;
    const long long first = live ? p + p / nz * 2 * nz : 0;
    // Row side: its row of U.
    const long long row = p0 + threadIdx.x / S::TPR;
    const bool rowLive = row < planes;
    const long long volume = (long long)nz * ny * M;  // complex pairs of one slot
    const V* vel = reinterpret_cast<const V*>(velocity) +
                   (rowLive ? ((row + row / nz * 2 * nz) * ny + y) * M : 0) + threadIdx.x % S::TPR;
    grid_wait();
    V sum[S::E];
#pragma unroll
    for (int e = 0; e < S::E; ++e) sum[e] = {T(0), T(0)};
    auto bins_of = [&](int f) {
        return reinterpret_cast<const V*>(in.data) + in.offset(first + (long long)f * nz) +
               in.planes * in.kxStride * y;
    };
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
        V v[S::E];
        const V* from = bins_of(f);
        if (f > 0) __syncthreads();  // the previous slot's exchange has been read
        // L2 prefetches, a 128-byte line each: this slot's velocity rows and, by the
        // first and last plane's threads, the next slot's bins.
        constexpr int kLine = phase_lanes<T>();
        if (rowLive)
            for (int e = int(threadIdx.x % S::TPR) * kLine; e < M; e += S::TPR * kLine)
                prefetch_l2(vel + f * volume + e - int(threadIdx.x % S::TPR));
        if (f < 2 && live && (threadIdx.x % S::B == 0 || threadIdx.x % S::B == S::B - 1)) {
            const V* next = bins_of(f + 1);
            for (int k = threadIdx.x / S::B; k < keep; k += S::TPR) prefetch_l2(next + in.planes * k);
        }
        V u[S::E];
        row_inverse<T, M>(v, data, from, in.planes, live, keep, twInverse, twFull, [&] {
#pragma unroll
            for (int e = 0; e < S::E; ++e) u[e] = rowLive ? __ldg(vel + f * volume + S::TPR * e) : V{T(0), T(0)};
        });
#pragma unroll
        for (int e = 0; e < S::E; ++e)
            sum[e] = f == 0 ? V{u[e].x * v[e].x, u[e].y * v[e].y}
                            : V{sum[e].x + u[e].x * v[e].x, sum[e].y + u[e].y * v[e].y};
    }
#pragma unroll
    for (int e = 0; e < S::E; ++e) sum[e] = {-scale * sum[e].x, -scale * sum[e].y};
    __syncthreads();
    V* out = reinterpret_cast<V*>(bins.data) + bins.offset(live ? p : 0) + bins.planes * bins.kxStride * y;
    row_forward<T, M>(sum, data, out, bins.planes, live, keep, twForward, twFull);
}

// Length-1 rows (Nx = 2): X[0] = x0 + x1, X[1] = x0 - x1.
template <typename T>
__global__ void rows_pair_kernel(int dir, int ny, long long planes, int keep, const T* __restrict__ realIn,
                                 T* __restrict__ realOut, DenseBins bins) {
    using V = cx<T>;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= planes * ny) return;
    const long long p = i % planes;
    const long long y = i / planes;
    V* b = reinterpret_cast<V*>(bins.data) + bins.offset(p);
    if (dir < 0) {
        const T x0 = realIn[(p * ny + y) * 2], x1 = realIn[(p * ny + y) * 2 + 1];
        b[bins.planes * (0 + bins.kxStride * y)] = {x0 + x1, T(0)};
        if (keep > 1) b[bins.planes * (1 + bins.kxStride * y)] = {x0 - x1, T(0)};
    } else {
        const T a = b[bins.planes * (0 + bins.kxStride * y)].x;
        const T c = keep > 1 ? b[bins.planes * (1 + bins.kxStride * y)].x : T(0);
        realOut[(p * ny + y) * 2] = a + c;
        realOut[(p * ny + y) * 2 + 1] = a - c;
    }
}

// The product stage for such rows.
template <typename T>
__global__ void rows_product_pair_kernel(int ny, int nz, long long planes, int keep, T scale,
                                         const T* __restrict__ velocity, DenseBins in, DenseBins bins) {
    using V = cx<T>;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= planes * ny) return;
    const long long p = i % planes;
    const long long y = i / planes;
    T s0 = T(0), s1 = T(0);
    for (int f = 0; f < 3; ++f) {
        const long long slot = p + p / nz * 2 * nz + (long long)f * nz;
        const V* b = reinterpret_cast<const V*>(in.data) + in.offset(slot) + in.planes * in.kxStride * y;
        const T a = b[0].x;
        const T c = keep > 1 ? b[in.planes].x : T(0);
        const T* u = velocity + (slot * ny + y) * 2;
        s0 += u[0] * (a + c);
        s1 += u[1] * (a - c);
    }
    V* b = reinterpret_cast<V*>(bins.data) + bins.offset(p) + bins.planes * bins.kxStride * y;
    b[0] = {-scale * s0 - scale * s1, T(0)};
    if (keep > 1) b[bins.planes] = {-scale * s0 + scale * s1, T(0)};
}

// ---------------------------------------------------------------------------
// Column transforms.  Grid (plane chunks, columns).

template <typename T>
__device__ __forceinline__ cx<T> view_load(const FieldView& v, long long mode, int z) {
    const long long i = z + v.modeStride * mode;
    if (v.im == nullptr) return reinterpret_cast<const cx<T>*>(v.re)[i];
    return {reinterpret_cast<const T*>(v.re)[i], reinterpret_cast<const T*>(v.im)[i]};
}

template <typename T>
__device__ __forceinline__ void view_store(const FieldView& v, long long mode, int z, cx<T> x) {
    const long long i = z + v.modeStride * mode;
    if (v.im == nullptr) {
        reinterpret_cast<cx<T>*>(v.re)[i] = x;
    } else {
        reinterpret_cast<T*>(v.re)[i] = x.x;
        reinterpret_cast<T*>(v.im)[i] = x.y;
    }
}

// Column kernels: tiles of one kx column of N points for B = L planes (128-byte
// pieces of every ky row); threads (plane b, t) with b fastest, so each
// exchange access is a run of L consecutive values, free of bank conflicts at
// any stride.  Elements go from HBM to registers and back: one exchange (two
// above 256 points) is the only shared-memory traffic.  Grid (plane chunks, kx).
// Bound: latency (load waits at 20-30 warps per SM), then HBM.  FP64: 512-point
// embedding / retention of 516 planes (1.1 GB) 436 / 358 -> 301 / 234 us, dense
// 256-point columns of 195 planes (205 MB) 49 -> 42 us; half as many planes
// per CTA moved the first two to 280 / 258 us, persistent CTAs to 329 / 289 us.
template <typename T, int N>
struct ColumnShape {
    using V = cx<T>;
    static constexpr int E = column_regs_per_thread(N, sizeof(T) == 8);
    static constexpr int TPC = N / E;
    static constexpr int B = phase_lanes<T>();
    static constexpr int NT = B * TPC;
    static constexpr size_t kBytes = TPC > 1 ? size_t(N) * B * sizeof(V) : 0;
    static constexpr int kCtas = resident_ctas<T>(NT, kBytes, E);
};

// Input and output of a column kernel: plane p of a dense bin array, or level
// p mod nz of retained view p / nz, so that chunks of planes run on across
// views and only the last one is ragged.
enum class ColumnIo { dense, views };

template <typename T, int N, int SIGN, ColumnIo IN, ColumnIo OUT>
__global__ void __launch_bounds__(ColumnShape<T, N>::NT, ColumnShape<T, N>::kCtas)
    columns_kernel(long long planes, DenseBins in, DenseBins out, int nz,
                   const __grid_constant__ ViewSet views, const int* __restrict__ cells, T scale,
                   const cx<T>* __restrict__ tw) {
    using V = cx<T>;
    using S = ColumnShape<T, N>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int b = threadIdx.x % S::B;
    const int t = threadIdx.x / S::B;
    PlaneExchange<V, S::B> xch{reinterpret_cast<V*>(smem_raw) + b};
    const long long kx = blockIdx.y;
    const long long p = (long long)blockIdx.x * S::B + b;
    const bool live = p < planes;
    FieldView view{};
    int z = 0;
    if (IN == ColumnIo::views || OUT == ColumnIo::views) {
        const int f = live ? int(p / nz) : 0;
        z = live ? int(p - (long long)f * nz) : 0;
        view = views.v[f];
    }
    const int* map = cells + kx * N + t;
    V v[S::E];
    if constexpr (IN == ColumnIo::views) {
        int cell[S::E];
#pragma unroll
        for (int e = 0; e < S::E; ++e) cell[e] = __ldg(map + S::TPC * e);
        grid_wait();
#pragma unroll
        for (int e = 0; e < S::E; ++e)
            v[e] = live && cell[e] >= 0 ? view_load<T>(view, cell[e] >> 1, z) : V{T(0), T(0)};
#pragma unroll
        for (int e = 0; e < S::E; ++e)
            if (cell[e] & 1) v[e] = cconj(v[e]);
    } else {
        grid_wait();
        const V* src =
            reinterpret_cast<const V*>(in.data) + in.offset(live ? p : 0) + in.planes * (kx + in.kxStride * t);
        const long long step = in.planes * in.kxStride * S::TPC;
#pragma unroll
        for (int e = 0; e < S::E; ++e) v[e] = live ? src[step * e] : V{T(0), T(0)};
    }
    fft_regs<T, N, S::E, SIGN>(v, t, tw, xch);
    if (!live) return;
    if constexpr (OUT == ColumnIo::views) {
#pragma unroll
        for (int e = 0; e < S::E; ++e) {
            const int cell = __ldg(map + S::TPC * e);
            if (cell < 0) continue;
            V x = cscale(v[e], scale);
            if (cell & 1) x = cconj(x);
            view_store<T>(view, cell >> 1, z, x);
        }
    } else {
        V* dst = reinterpret_cast<V*>(out.data) + out.offset(p) + out.planes * (kx + out.kxStride * t);
        const long long step = out.planes * out.kxStride * S::TPC;
#pragma unroll
        for (int e = 0; e < S::E; ++e) dst[step * e] = v[e];
    }
}

// Plain retention from a dense spectrum: one thread per (mode, z) of a view.
template <typename T>
__global__ void gather_dense_kernel(int nz, long long modes, const int* __restrict__ modeKx,
                                    const int* __restrict__ modeKy, const unsigned char* __restrict__ modeConj,
                                    DenseBins in, ViewSet views, T scale) {
    using V = cx<T>;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int f = blockIdx.y;
    if (i >= modes * nz) return;
    const int z = int(i % nz);
    const long long m = i / nz;
    const V* src = reinterpret_cast<const V*>(in.data);
    V v = src[(long long)f * nz + z + in.planes * ((long long)__ldg(modeKx + m) + in.kxStride * __ldg(modeKy + m))];
    v = cscale(v, scale);
    if (__ldg(modeConj + m)) v = cconj(v);
    view_store<T>(views.v[f], m, z, v);
}

// Plain embedding into a dense spectrum: every cell of the column band is
// written (zero where no mode lands), so no separate clear is needed.
template <typename T>
__global__ void embed_dense_kernel(int ny, int nz, ViewSet views, ModeTables tables, DenseBins out) {
    using V = cx<T>;
    const int f = blockIdx.z;
    const int kx = blockIdx.y;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)ny * nz) return;
    const int z = int(i % nz);
    const int ky = int(i / nz);
    const int e = __ldg(tables.cellMap + (long long)kx * ny + ky);
    V v = {T(0), T(0)};
    if (e >= 0) {
        v = view_load<T>(views.v[f], e >> 1, z);
        if (e & 1) v = cconj(v);
    }
    reinterpret_cast<V*>(out.data)[(long long)f * nz + z + out.planes * ((long long)kx + out.kxStride * ky)] = v;
}

// ---------------------------------------------------------------------------
// Dispatch helpers.

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

#define SKB_LENGTH_CASE(n, ...) \
    case n: {                   \
        constexpr int L = n;    \
        __VA_ARGS__;            \
    } break;
// Half row lengths (Nx / 2) up to 512; column lengths reach 1024.
#define SKB_HALF_CASES(...)         \
    SKB_LENGTH_CASE(2, __VA_ARGS__)   \
    SKB_LENGTH_CASE(4, __VA_ARGS__)   \
    SKB_LENGTH_CASE(8, __VA_ARGS__)   \
    SKB_LENGTH_CASE(16, __VA_ARGS__)  \
    SKB_LENGTH_CASE(32, __VA_ARGS__)  \
    SKB_LENGTH_CASE(64, __VA_ARGS__)  \
    SKB_LENGTH_CASE(128, __VA_ARGS__) \
    SKB_LENGTH_CASE(256, __VA_ARGS__) \
    SKB_LENGTH_CASE(512, __VA_ARGS__)
#define SKB_HALF_SWITCH(n, ...)                   \
    switch (n) {                                  \
        SKB_HALF_CASES(__VA_ARGS__)               \
        default: return cudaErrorInvalidValue;    \
    }
#define SKB_LENGTH_SWITCH(n, ...)                 \
    switch (n) {                                  \
        SKB_HALF_CASES(__VA_ARGS__)               \
        SKB_LENGTH_CASE(1024, __VA_ARGS__)        \
        default: return cudaErrorInvalidValue;    \
    }

template <typename T>
cudaError_t rows_forward_t(int nx, int ny, long long planes, int keep, const void* real, DenseBins bins,
                           const void* twHalf, const void* twFull, cudaStream_t stream) {
    const int M = nx / 2;
    if (M == 1) {
        const long long n = planes * ny;
        rows_pair_kernel<T><<<unsigned((n + 255) / 256), 256, 0, stream>>>(-1, ny, planes, keep,
                                                                            static_cast<const T*>(real), nullptr, bins);
        return cudaGetLastError();
    }
    SKB_HALF_SWITCH(M, {
        using S = RowShape<T, L>;
        auto kernel = rows_forward_kernel<T, L>;
        const cudaError_t err = allow_smem(kernel, S::kBytes);
        if (err != cudaSuccess) return err;
        const dim3 grid(unsigned((planes + S::B - 1) / S::B), unsigned(ny));
        return launch_chained(kernel, grid, S::NT, S::kBytes, stream, ny, planes, keep, static_cast<const T*>(real),
                              bins, static_cast<const cx<T>*>(twHalf), static_cast<const cx<T>*>(twFull));
    });
    return cudaGetLastError();
}

template <typename T>
cudaError_t rows_inverse_t(int nx, int ny, long long planes, int keep, DenseBins bins, void* real,
                           const void* twHalf, const void* twFull, cudaStream_t stream) {
    const int M = nx / 2;
    if (M == 1) {
        const long long n = planes * ny;
        rows_pair_kernel<T><<<unsigned((n + 255) / 256), 256, 0, stream>>>(+1, ny, planes, keep, nullptr,
                                                                            static_cast<T*>(real), bins);
        return cudaGetLastError();
    }
    SKB_HALF_SWITCH(M, {
        using S = RowShape<T, L>;
        auto kernel = rows_inverse_kernel<T, L>;
        const cudaError_t err = allow_smem(kernel, S::kBytes);
        if (err != cudaSuccess) return err;
        const dim3 grid(unsigned((planes + S::B - 1) / S::B), unsigned(ny));
        return launch_chained(kernel, grid, S::NT, S::kBytes, stream, ny, planes, keep, bins, static_cast<T*>(real),
                              static_cast<const cx<T>*>(twHalf), static_cast<const cx<T>*>(twFull));
    });
    return cudaGetLastError();
}

template <typename T>
cudaError_t rows_product_t(int nx, int ny, int nz, long long planes, int keep, double scale, const void* velocity,
                           DenseBins in, DenseBins out, const void* twInverse, const void* twForward,
                           const void* twFull, cudaStream_t stream) {
    if (nx == 2) {
        const long long n = planes * ny;
        rows_product_pair_kernel<T><<<unsigned((n + 255) / 256), 256, 0, stream>>>(
            ny, nz, planes, keep, T(scale), static_cast<const T*>(velocity), in, out);
        return cudaGetLastError();
    }
    SKB_HALF_SWITCH(nx / 2, {
        using S = RowShape<T, L>;
        auto kernel = rows_product_kernel<T, L>;
        const cudaError_t err = allow_smem(kernel, S::kBytes);
        if (err != cudaSuccess) return err;
        const dim3 grid(unsigned((planes + S::B - 1) / S::B), unsigned(ny));
        return launch_chained(kernel, grid, S::NT, S::kBytes, stream, ny, nz, planes, keep, T(scale),
                              static_cast<const T*>(velocity), in, out, static_cast<const cx<T>*>(twInverse),
                              static_cast<const cx<T>*>(twForward), static_cast<const cx<T>*>(twFull));
    });
    return cudaGetLastError();
}

template <typename T, int SIGN, ColumnIo IN, ColumnIo OUT>
cudaError_t columns_t(int ny, int columns, long long planes, DenseBins in, DenseBins out, int nz, const ViewSet& views,
                      const int* cells, double scale, const void* tw, cudaStream_t stream) {
    SKB_LENGTH_SWITCH(ny, {
        using S = ColumnShape<T, L>;
        auto kernel = columns_kernel<T, L, SIGN, IN, OUT>;
        const cudaError_t err = allow_smem(kernel, S::kBytes);
        if (err != cudaSuccess) return err;
        const dim3 grid(unsigned((planes + S::B - 1) / S::B), unsigned(columns));
        return launch_chained(kernel, grid, S::NT, S::kBytes, stream, planes, in, out, nz, views, cells, T(scale),
                              static_cast<const cx<T>*>(tw));
    });
    return cudaGetLastError();
}

const ViewSet kNoViews{};

}  // namespace

bool supported_length(long long n) { return n >= 2 && n <= 1024 && (n & (n - 1)) == 0; }

cudaError_t launch_rows_forward(Precision p, int nx, int ny, long long planes, int keep, const void* real,
                                DenseBins bins, const void* twHalf, const void* twFull, cudaStream_t stream) {
    if (planes <= 0) return cudaSuccess;
    return p == Precision::f64 ? rows_forward_t<double>(nx, ny, planes, keep, real, bins, twHalf, twFull, stream)
                               : rows_forward_t<float>(nx, ny, planes, keep, real, bins, twHalf, twFull, stream);
}

cudaError_t launch_rows_inverse(Precision p, int nx, int ny, long long planes, int keep, DenseBins bins, void* real,
                                const void* twHalf, const void* twFull, cudaStream_t stream) {
    if (planes <= 0) return cudaSuccess;
    return p == Precision::f64 ? rows_inverse_t<double>(nx, ny, planes, keep, bins, real, twHalf, twFull, stream)
                               : rows_inverse_t<float>(nx, ny, planes, keep, bins, real, twHalf, twFull, stream);
}

cudaError_t launch_rows_product(Precision p, int nx, int ny, int nz, int members, int keep, double scale,
                                const void* velocity, DenseBins in, DenseBins out, const void* twInverse,
                                const void* twForward, const void* twFull, cudaStream_t stream) {
    const long long planes = (long long)members * nz;
    if (planes <= 0) return cudaSuccess;
    return p == Precision::f64 ? rows_product_t<double>(nx, ny, nz, planes, keep, scale, velocity, in, out, twInverse,
                                                        twForward, twFull, stream)
                               : rows_product_t<float>(nx, ny, nz, planes, keep, scale, velocity, in, out, twInverse,
                                                       twForward, twFull, stream);
}

cudaError_t launch_columns_dense(Precision p, int sign, int ny, int columns, long long planes, DenseBins in,
                                 DenseBins out, const void* tw, cudaStream_t stream) {
    if (planes <= 0 || columns <= 0) return cudaSuccess;
    constexpr auto D = ColumnIo::dense;
    if (p == Precision::f64)
        return sign < 0 ? columns_t<double, -1, D, D>(ny, columns, planes, in, out, 1, kNoViews, nullptr, 1.0, tw, stream)
                        : columns_t<double, +1, D, D>(ny, columns, planes, in, out, 1, kNoViews, nullptr, 1.0, tw, stream);
    return sign < 0 ? columns_t<float, -1, D, D>(ny, columns, planes, in, out, 1, kNoViews, nullptr, 1.0, tw, stream)
                    : columns_t<float, +1, D, D>(ny, columns, planes, in, out, 1, kNoViews, nullptr, 1.0, tw, stream);
}

cudaError_t launch_columns_embed(Precision p, int ny, int nz, int columns, const ViewSet& views,
                                 const ModeTables& tables, DenseBins out, const void* tw, cudaStream_t stream) {
    if (views.count <= 0 || columns <= 0) return cudaSuccess;
    constexpr auto D = ColumnIo::dense, W = ColumnIo::views;
    const long long planes = (long long)nz * views.count;
    return p == Precision::f64
               ? columns_t<double, +1, W, D>(ny, columns, planes, {}, out, nz, views, tables.cellMap, 1.0, tw, stream)
               : columns_t<float, +1, W, D>(ny, columns, planes, {}, out, nz, views, tables.cellMap, 1.0, tw, stream);
}

cudaError_t launch_columns_gather(Precision p, int ny, int nz, int columns, DenseBins in, const ViewSet& views,
                                  const ModeTables& tables, double scale, const void* tw, cudaStream_t stream) {
    if (views.count <= 0 || columns <= 0) return cudaSuccess;
    constexpr auto D = ColumnIo::dense, W = ColumnIo::views;
    const long long planes = (long long)nz * views.count;
    return p == Precision::f64
               ? columns_t<double, -1, D, W>(ny, columns, planes, in, {}, nz, views, tables.gatherMap, scale, tw, stream)
               : columns_t<float, -1, D, W>(ny, columns, planes, in, {}, nz, views, tables.gatherMap, scale, tw, stream);
}

cudaError_t launch_gather_dense(Precision p, int ny, int nz, long long modes, const int* modeKx, const int* modeKy,
                                const unsigned char* modeConj, DenseBins in, const ViewSet& views, double scale,
                                cudaStream_t stream) {
    (void)ny;
    if (modes <= 0 || views.count <= 0) return cudaSuccess;
    const long long n = modes * nz;
    dim3 grid(unsigned((n + 255) / 256), unsigned(views.count));
    if (p == Precision::f64)
        gather_dense_kernel<double><<<grid, 256, 0, stream>>>(nz, modes, modeKx, modeKy, modeConj, in, views, scale);
    else
        gather_dense_kernel<float><<<grid, 256, 0, stream>>>(nz, modes, modeKx, modeKy, modeConj, in, views,
                                                             float(scale));
    return cudaGetLastError();
}

cudaError_t launch_embed_dense(Precision p, int ny, int nz, int columns, const ViewSet& views,
                               const ModeTables& tables, DenseBins out, cudaStream_t stream) {
    if (views.count <= 0 || columns <= 0) return cudaSuccess;
    const long long n = (long long)ny * nz;
    dim3 grid(unsigned((n + 255) / 256), unsigned(columns), unsigned(views.count));
    if (p == Precision::f64)
        embed_dense_kernel<double><<<grid, 256, 0, stream>>>(ny, nz, views, tables, out);
    else
        embed_dense_kernel<float><<<grid, 256, 0, stream>>>(ny, nz, views, tables, out);
    return cudaGetLastError();
}

}  // namespace skb
