// Fused row stage of the split-precision flux (FP32).
//
// One CTA owns one row y of B consecutive z-planes of one ensemble member and
// does, entirely on chip, what the staged path spreads over a row kernel for U, V and
// W and one per target, with three real volumes (benchmark.cpp:4405-4424 order):
//   U,V,W rows      <- c2r of the column-transformed bins of input slots 0..2,
//                      kept in registers;
//   for each target t:
//     q_t,x/y/z rows <- c2r of slots 3+3t .. 5+3t;
//     target row     = -scale*(u*q_x + v*q_y + w*q_z)   (pointwise_advection.cpp:143-147)
//     target bins    <- r2c of the target row, kx < keep.
// The c2r / r2c are the same half-length complex FFT formulation as the
// staged row kernels (horizontal.cu), so both paths share their numerics.
// Two kernels: 128-, 256- and 512-point rows run several planes per warp
// (rows_flux_pair_kernel, below); in the other, for 64-point rows and as a choice of
// the autotuner at 512 points, each warp owns one z-plane and transforms it with
// warp-synchronous passes
// (warp_fft; for 512-point rows warp_fft_rr, whose first and last passes work
// in registers); every lane keeps the same Nx/64 x-pairs of its plane across
// all transforms, which is what lets U,V,W and the product stay in registers.
// The 3+3T slots are consumed in order, so the bins of slot f+1 are copied
// into a second shared stage with cp.async while slot f is transformed; the
// only CTA-wide barriers are one per slot and one per target.
// Each stage row holds kx = 0..M and is zero beyond keep (written once, never
// copied over), so the c2r pre-processing reads bins k and M-k without range
// tests; the r2c twiddles and the 512-point FFT's lane-ordered twiddle table
// are copied into shared memory once per CTA.

#include "flux_rows.hpp"

#include "async_copy.cuh"
#include "fft_regs.cuh"
#include "launch.cuh"
#include "tensor_map.hpp"

namespace skb {
namespace {

// Per-warp padded sequence region (pad16 of the largest index, plus slack).
template <int M>
constexpr int region() {
    return M + M / 16 + 8;
}
// Stage row stride: kx = 0..M, and a residue mod 16 (in 8-byte words) that
// spreads one cp.async instruction's B planes x 32/B consecutive kx over the
// 16 bank pairs exactly twice (4 for B = 4 and 8, 1 for B = 16).
template <int M, int B>
constexpr int stage_row() {
    constexpr int want = B == 16 ? 1 : 4;
    return M + 1 + ((want - (M + 1) % 16) + 16) % 16;
}
// Output tile [k][b], row stride B, plane b of row k at b ^ swz(k): a warp's
// 16 consecutive kx of one plane and a copy-out instruction's B planes x 32/B
// consecutive kx both touch every bank pair equally often.
// B = 24 (no XOR swizzle stays inside a 24-plane row): rows of 25 slots,
// whose odd stride spreads 16 consecutive kx of one plane over all bank pairs.
template <int B>
constexpr int out_row() {
    return B == 24 ? 25 : B;
}
template <int B>
__device__ __forceinline__ int out_slot(int k, int b) {
    if constexpr (B == 24)
        return k * out_row<B>() + b;
    else
        return k * B + (b ^ ((k / (16 / B)) & (B - 1)));
}
// Entries of the lane-ordered FFT twiddle table (512-point rows only).
template <int M>
constexpr int rr_entries() {
    if constexpr (M == 256) {
        return rr_table_size<M>();
    } else {
        return 0;
    }
}
template <int M, int B>
constexpr size_t rows_smem_words(int keep) {
    return size_t(B) * region<M>() + 2 * size_t(B) * stage_row<M, B>() + size_t(keep) * B + M + rr_entries<M>();
}

// Launch bounds keep 128 registers per thread whatever the CTA width:
// 16 / B CTAs of 32 * B threads fill 512 threads' worth of the register file.
template <int M, int B>
__global__ void __launch_bounds__(32 * B, 16 / B) rows_flux_kernel(RowFluxArgs a) {
    using V = float2;
    constexpr int NT = 32 * B;
    constexpr int PER = M / 32;  // elements of its plane each lane keeps in registers
    constexpr int XP = region<M>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int KP = stage_row<M, B>();
    static_assert(M != 256 || XP >= rr_region_min<256>(), "plane region too small for warp_fft_rr");
    const int keep = a.keep;
    V* xs = reinterpret_cast<V*>(smem_raw);
    V* stage0 = xs + B * XP;
    V* stage1 = stage0 + B * KP;
    V* outTile = stage1 + B * KP;  // [k][b] at out_slot(k, b)
    V* tf = outTile + keep * B;        // twFull[0..M)
    V* tt = tf + M;                    // warp_fft_rr table (M = 256)
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int zChunks = (a.nz + B - 1) / B;
    const int member = blockIdx.x / zChunks;
    const int z0 = (blockIdx.x % zChunks) * B;
    const int y = blockIdx.y;
    const V* twHalf = static_cast<const V*>(a.twHalf);
    const V* twFull = static_cast<const V*>(a.twFull);
    const V* in = static_cast<const V*>(a.binsIn.data);
    V* out = static_cast<V*>(a.binsOut.data);
    const long long inRow = a.binsIn.planes;  // stride between kx
    const long long outRow = a.binsOut.planes;
    V* x = xs + warp * XP;  // this warp's plane

    for (int i = tid; i < M; i += NT) tf[i] = twFull[i];
    if constexpr (rr_entries<M>() > 0) rr_fill_table<float, M>(tt, twHalf, tid, NT);
    for (int i = tid; i < 2 * B * (KP - keep); i += NT) {
        const int row = i / (KP - keep);
        stage0[row * KP + keep + i % (KP - keep)] = V{0.f, 0.f};
    }

    // Asynchronous copy of slot f's bins of this row into a plane-major stage
    // [b][k]; consecutive threads read consecutive planes of one kx (the
    // planes-innermost global rows), planes beyond Nz are zero-filled.  NT is a
    // multiple of B, so a thread keeps its plane cb and steps kx by NT / B.
    constexpr int KSTEP = NT / B;
    const int cb = tid % B;
    const int ck = tid / B;
    const bool cok = z0 + cb < a.nz;
    auto issue = [&](int f, V* stage) {
        const long long plane = (static_cast<long long>(member) * a.fieldsIn + f) * a.zStride + z0 + cb;
        const V* src = in + plane + inRow * (a.binsIn.kxStride * y + ck);
        V* dst = stage + cb * KP + ck;
        for (int k = ck; k < keep; k += KSTEP, src += inRow * KSTEP, dst += KSTEP) cp_async8(dst, cok ? src : in, cok ? 8 : 0);
        cp_async_commit();
    };

    // Inverse row transform of slot f into this lane's registers r[]: element
    // lane + 32e of the warp's plane.
    auto inverse_row = [&](int f, V (&r)[PER]) {
        cp_async_wait_all();
        __syncthreads();
        if (f + 1 < a.fieldsIn) issue(f + 1, ((f + 1) & 1) ? stage1 : stage0);
        const V* st = ((f & 1) ? stage1 : stage0) + warp * KP;
        auto load = [&](int k) -> V {
            if (k >= keep) return V{0.f, 0.f};
            V v = st[k];
            if (k == 0 || k == M) v.y = 0.f;
            return v;
        };
        if constexpr (M == 256) {
            // Pre-processed half-length spectrum straight into registers
            // (element k = lane + 32e), then the register-ended FFT.  At k = 0
            // (lane 0, e = 0) the bins 0 and M are real, and the general form
            // reduces to {X0 + XM, X0 - XM} since tf[0] = 1.
            const V* stk = st + lane;
            const V* stm = st + (M - lane);
            const V* tfk = tf + lane;
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                V xk = stk[32 * e];
                V xm = stm[-32 * e];
                if (e == 0 && lane == 0) {
                    xk.y = 0.f;
                    xm.y = 0.f;
                }
                const V s = cadd(xk, cconj(xm));
                const V d = csub(xk, cconj(xm));
                const V t = cmulc(d, tfk[32 * e]);
                r[e] = {s.x - t.y, s.y + t.x};
            }
            warp_fft_rr<float, M, +1>(r, x, tt, lane);
        } else {
            constexpr int pairs = M / 2 + 1;
            for (int k = lane; k < pairs; k += 32) {
                if (k == 0) {
                    const V x0 = load(0);
                    const V xm = load(M);
                    x[pad16(0)] = {x0.x + xm.x, x0.x - xm.x};
                    continue;
                }
                const int kk = M - k;
                const V xk = load(k);
                const V xm = load(kk);
                {
                    const V s = cadd(xk, cconj(xm));
                    const V d = csub(xk, cconj(xm));
                    const V t = cmulc(d, tf[k]);
                    x[pad16(k)] = {s.x - t.y, s.y + t.x};
                }
                if (kk != k) {
                    const V s = cadd(xm, cconj(xk));
                    const V d = csub(xm, cconj(xk));
                    const V t = cmulc(d, tf[kk]);
                    x[pad16(kk)] = {s.x - t.y, s.y + t.x};
                }
            }
            __syncwarp();
            warp_fft<float, M, +1>(x, twHalf, lane);
#pragma unroll
            for (int e = 0; e < PER; ++e) r[e] = x[pad16(lane + 32 * e)];
            __syncwarp();
        }
    };

    issue(0, stage0);
    V u[PER], v[PER], w[PER];
    inverse_row(0, u);
    inverse_row(1, v);
    inverse_row(2, w);
    const float scale = a.scale;
    for (int t = 0; t < a.targets; ++t) {
        V acc[PER], q[PER];
        inverse_row(3 + 3 * t, q);
#pragma unroll
        for (int e = 0; e < PER; ++e) acc[e] = {u[e].x * q[e].x, u[e].y * q[e].y};
        inverse_row(4 + 3 * t, q);
#pragma unroll
        for (int e = 0; e < PER; ++e) acc[e] = {acc[e].x + v[e].x * q[e].x, acc[e].y + v[e].y * q[e].y};
        inverse_row(5 + 3 * t, q);
#pragma unroll
        for (int e = 0; e < PER; ++e)
            acc[e] = {-scale * (acc[e].x + w[e].x * q[e].x), -scale * (acc[e].y + w[e].y * q[e].y)};
        if constexpr (M == 256) {
            warp_fft_rr<float, M, -1>(acc, x, tt, lane);
            // pad16(lane + 32e) = lane + lane/16 + 34e
            V* o = x + lane + (lane >> 4);
#pragma unroll
            for (int e = 0; e < PER; ++e) o[34 * e] = acc[e];
        } else {
#pragma unroll
            for (int e = 0; e < PER; ++e) x[pad16(lane + 32 * e)] = acc[e];
            __syncwarp();
            warp_fft<float, M, -1>(x, twHalf, lane);
        }
        __syncwarp();
        // Real-spectrum split of the half-length FFT, kx < keep, into [k][b].
        const V zz = x[pad16(0)];
        for (int k = lane; k < keep; k += 32) {
            V X;
            if (k == 0) {
                X = {zz.x + zz.y, 0.f};
            } else if (k == M) {
                X = {zz.x - zz.y, 0.f};
            } else {
                const V zk = x[pad16(k)];
                const V zm = cconj(x[pad16(M - k)]);
                const V ev = cscale(cadd(zk, zm), 0.5f);
                const V d = csub(zk, zm);
                const V o = {0.5f * d.y, -0.5f * d.x};
                X = cadd(ev, cmul(tf[k], o));
            }
            outTile[out_slot<B>(k, warp)] = X;
        }
        __syncthreads();
        // Coalesced rows of B planes per kx.
        if (cok) {
            const long long plane = (static_cast<long long>(member) * a.targets + t) * a.zStride + z0 + cb;
            V* dst = out + plane + outRow * (a.binsOut.kxStride * y + ck);
            for (int k = ck; k < keep; k += KSTEP, dst += outRow * KSTEP) *dst = outTile[out_slot<B>(k, cb)];
        }
        // The next outTile write happens after the next inverse_row's barrier.
    }
}

// ---------------------------------------------------------------------------
// 512-point rows, two planes per warp, and 256- and 128-point rows with four and
// eight (T = 8 and 4 lanes per plane, the second radix 8 and 4).
//
// The 256-point complex FFT of the half-length formulation is split 16 x 16:
// lane t of a half-warp holds elements t + 16 m (m = 0..15) of its plane's
// sequence; a radix-16 DFT over m in registers, the twiddles W256^(t k2), one
// 16 x 16 transpose through shared memory, and a second radix-16 DFT in
// registers leave output k = t + 16 k1 in register k1 — the same lane-owned
// positions as the input, so U, V, W and the product stay in registers across
// all transforms as in the warp-per-plane kernel, with one shared-memory
// exchange per transform instead of two.  Warp w owns planes 2w and 2w + 1.

constexpr int kPairM = 256;  // half-length of the 512-point rows
// An 8-byte shared access is served half-warp by half-warp, and the 16 lanes of one
// touch each of the 16 bank pairs once if they are 8 consecutive bins of two adjacent
// planes (T = M/16 lanes per plane: 16 or 8) or 4 bins of the planes p, p + 1, p + B/2,
// p + B/2 + 1 (T = 4): so lie the lanes in the TMA forms.  512-point rows with 16 bins
// of one plane per half-warp, as the cp.async forms' [plane][bin] stages want them,
// read the swizzled stages with every second access repeated: 5844 -> 5412 us for 8
// members at Nz 129.
//
// Exchange words per plane: one spare per 16 makes the first pass's stride-16 stores
// conflict-free, and the region's length (8 or 4 mod 16) keeps a half-warp's two or
// four planes apart.
constexpr int pair_xch(int M, bool interleaved) { return M + M / 16 + (interleaved ? 8 : 0); }
// Output tile of the TMA forms, [k][b] like out_slot, for those half-warps.
template <int B>
__device__ __forceinline__ int pair_out_slot(int k, int b) {
    return k * B + (b ^ ((B == 16 ? k & 7 : (k >> 1) & 3) << 1));
}
// Bins the pre-processing reads: the 2/3 rule keeps kx < 11 T (T = M/16 lanes
// per plane; 171 of 176, 86 of 88, 43 of 44), so bins k >= 11 T and, with them,
// the products of registers m >= 11 (k) and m <= 4 (M - k) are left out.
constexpr int pair_keep(int M) { return 11 * (M / 16); }

// A plane's exchange among its lanes.
struct PairExchange {
    float2* x;
    __device__ __forceinline__ void store(int i, float2 v) { x[i + (i >> 4)] = v; }
    __device__ __forceinline__ float2 load(int i) const { return x[i + (i >> 4)]; }
    __device__ __forceinline__ void fence() const { __syncwarp(); }
};
template <int B>
constexpr int pair_stage_row() {
    // kx = 0..M (the pre-processing reads X[M - k]), and a residue mod 16 (in
    // 8-byte words) that spreads one cp.async instruction's B planes x 32/B
    // kx over the 16 bank pairs exactly twice.
    // (B = 24: an odd stride, at most three accesses per bank pair.)
    constexpr int want = B == 16 || B == 24 ? 1 : 2;
    return kPairM + 1 + ((want - (kPairM + 1) % 16) + 16) % 16;
}
template <int B>
constexpr size_t pair_smem_words(int keep) {
    return 2 * size_t(B) * pair_stage_row<B>() + size_t(B) * pair_xch(kPairM, false) + size_t(keep) * out_row<B>() + kPairM +
           kPairM;
}

// TMA form of the stage: rows kx = 0..pair_keep(M) (the pre-processing reads
// no bin beyond, see inverse_row), each row the B planes' values
// (64 or 128 bytes) in the SWIZZLE_64B / SWIZZLE_128B pattern the tensor
// copy writes; rows keep..pair_keep(M) are zero.  Stages start on 1024-byte
// boundaries (the swizzle pattern's period).
template <int M, int B>
constexpr size_t tma_stage_bytes() {
    return (size_t(pair_keep(M) + 1) * B * 8 + 1023) / 1024 * 1024;
}
// The third velocity row W is kept in a lane-private shared region (16 values
// per thread) instead of registers in the forms compiled for 12 warps per SM.
template <int M, int B, int MINB, int NS>
constexpr bool pair_w_in_smem() {
    return NS == 2 && MINB * M * B == 3 * 256 * 8;
}
template <int M, int B, int NS, bool WSM>
constexpr size_t pair_tma_smem_bytes(int keep) {
    return 1024 + NS * tma_stage_bytes<M, B>() +
           sizeof(float2) * (size_t(B) * pair_xch(M, M == kPairM) + size_t(keep) * out_row<B>() + M + M +
                             (WSM ? size_t(M) * B : 0));
}
// Byte offset of (kx k, plane b) in a swizzled TMA stage.
template <int B>
__device__ __forceinline__ unsigned tma_stage_offset(int k, int b) {
    const unsigned off = static_cast<unsigned>((k * B + b) * 8);
    return off ^ (((off >> 7) & (B == 8 ? 3u : 7u)) << 4);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// A bounded wait on an mbarrier phase (false once the limit is reached).
__device__ __forceinline__ bool stage_wait(unsigned bar, unsigned parity, long long limit = 1LL << 22) {
    for (long long i = 0; i < limit; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// MINB: resident CTAs per SM the register allocation must allow (2 for B = 8,
// 1 for B = 16: about 240 registers; 3 for the B = 8 form that trades spills
// to L1-cached local memory for occupancy).
// TMA (NS = 2 or 3 stages; 0: cp.async): each slot's stage is filled by one
// tensor copy (thread 0, onto an mbarrier; `tmIn` maps the input bins as
// [cell][plane]) instead of 8-byte cp.async by every thread, NS - 1 slots
// ahead of the one being transformed.  Thread 0's bounded wait on the copy is
// folded into the slot's CTA barrier (__syncthreads_and), so an expired wait
// makes every thread leave together after setting the error word.
template <int M, int B, int MINB, int NS>
__global__ void __launch_bounds__(M / 16 * B, MINB)
    rows_flux_pair_kernel(RowFluxArgs a, const __grid_constant__ CUtensorMap tmIn) {
    using V = float2;
    constexpr bool TMA = NS != 0;
    constexpr int NST = TMA ? NS : 2;  // stages
    constexpr int T = M / 16;  // lanes per plane
    constexpr int NT = T * B;
    constexpr int KP = pair_stage_row<B>();
    constexpr bool PAIRED = TMA && T == 16;  // lanes 2 t and 2 t + 1 hold a warp's two planes
    constexpr int XCH = pair_xch(M, PAIRED);
    static_assert(M == kPairM || TMA, "the cp.async stages are laid out for 512-point rows");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long stageFull[NST];
    __shared__ __align__(8) unsigned long long never;  // nothing arrives on it (expired-wait test)
    const int keep = a.keep;
    unsigned char* tmaBase =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    auto stage_of = [&](int f) -> V* {
        if constexpr (TMA)
            return reinterpret_cast<V*>(tmaBase + (f % NST) * tma_stage_bytes<M, B>());
        else
            return reinterpret_cast<V*>(smem_raw) + (f & 1) * B * KP;
    };
    V* stage0 = stage_of(0);
    V* xchAll = TMA ? reinterpret_cast<V*>(tmaBase + NST * tma_stage_bytes<M, B>()) : stage0 + 2 * B * KP;
    V* outTile = xchAll + B * XCH;          // [k][b] at outSlot(k, b)
    V* tf = outTile + keep * out_row<B>();  // twFull[0..M)
    V* tw2 = tf + M;                     // fft_regs' table: tw2[16 (r - 1) + j] = twHalf[j r]
    // Two-stage TMA forms at 12 warps per SM: W (16 values per thread) lives
    // here, at wsm[e * NT + tid], which takes the register peak of u, v, w, the
    // product and the current derivative under the 168-register bound.
    constexpr bool WSM = pair_w_in_smem<M, B, MINB, NS>();
    V* wsm = tw2 + M;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    // These lanes' exchange region and plane within the CTA.
    const int t = PAIRED ? lane >> 1 : tid % T;
    const int region = PAIRED ? 2 * (tid >> 5) + (lane & 1) : tid / T;
    const int pl = T == 4 ? (region & 1) | (region & 2) * (B / 4) | (region >> 2) << 1 : region;
    auto outSlot = [](int k, int b) { return TMA ? pair_out_slot<B>(k, b) : out_slot<B>(k, b); };
    const int zChunks = (a.nz + B - 1) / B;
    const int member = blockIdx.x / zChunks;
    const int z0 = (blockIdx.x % zChunks) * B;
    const int y = blockIdx.y;
    const V* twHalf = static_cast<const V*>(a.twHalf);
    const V* twFull = static_cast<const V*>(a.twFull);
    const V* in = static_cast<const V*>(a.binsIn.data);
    V* out = static_cast<V*>(a.binsOut.data);
    const long long inRow = a.binsIn.planes;
    const long long outRow = a.binsOut.planes;
    PairExchange xch{xchAll + region * XCH};

    for (int i = tid; i < M; i += NT) {
        tf[i] = twFull[i];
        if (i < M - 16) tw2[i] = twHalf[(i & 15) * ((i >> 4) + 1)];
    }
    if constexpr (TMA) {
        // Rows keep..pair_keep(M) of every stage are zero (the tensor copies
        // write rows 0..keep-1 only; the swizzle stays inside a row).
        const int zeros = (pair_keep(M) + 1 - keep) * B;
        for (int i = tid; i < NST * zeros; i += NT) {
            const int st = i / zeros;
            reinterpret_cast<V*>(tmaBase + st * tma_stage_bytes<M, B>())[keep * B + i - st * zeros] = V{0.f, 0.f};
        }
        if (tid == 0) {
            for (int i = 0; i < NST; ++i)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&stageFull[i])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&never)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    } else {
        for (int i = tid; i < 2 * B * (KP - keep); i += NT) {
            const int row = i / (KP - keep);
            stage0[row * KP + keep + i % (KP - keep)] = V{0.f, 0.f};
        }
    }

    // Slot f's bins of this row into a plane-major stage [b][k] (cp.async, as
    // in the warp-per-plane kernel; planes beyond Nz are zero-filled), or, in
    // the TMA form, into a swizzled [k][b] stage by one tensor copy (planes
    // beyond Nz then hold the next slot's or padding values; those planes'
    // results are never stored).
    constexpr int KSTEP = NT / B;
    const int cb = tid % B;
    const int ck = tid / B;
    const bool cok = z0 + cb < a.nz;
    // This lane's byte offsets of bins t and M - t; the swizzle repeats every 8
    // rows, so with fewer than 8 lanes per plane register m = 1 has its own.
    constexpr int PER = T < 8 ? 8 / T : 1;
    int tmaLo[PER], tmaHi[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        tmaLo[i] = static_cast<int>(tma_stage_offset<B>(t + T * i, pl));
        tmaHi[i] = static_cast<int>(tma_stage_offset<B>(M - t - T * i, pl));
    }
    auto issue = [&](int f) {
        V* stage = stage_of(f);
        if constexpr (TMA) {
            if (tid == 0) {
                const int x = (member * a.fieldsIn + f) * a.zStride + z0;
                const int yc = static_cast<int>(a.binsIn.kxStride * y);
                const unsigned bar = smem_addr(&stageFull[f % NST]);
                // The stage's earlier shared-memory reads precede the copy's writes.
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"(static_cast<unsigned>(keep * B * 8))
                             : "memory");
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                    "%3}], [%4];" ::"r"(smem_addr(stage)),
                    "l"(reinterpret_cast<unsigned long long>(&tmIn)), "r"(x), "r"(yc), "r"(bar)
                    : "memory");
            }
        } else {
            const long long plane = (static_cast<long long>(member) * a.fieldsIn + f) * a.zStride + z0 + cb;
            const V* src = in + plane + inRow * (a.binsIn.kxStride * y + ck);
            V* dst = stage + cb * KP + ck;
            for (int k = ck; k < keep; k += KSTEP, src += inRow * KSTEP, dst += KSTEP) cp_async8(dst, cok ? src : in, cok ? 8 : 0);
            cp_async_commit();
        }
    };

    // c2r of slot f into r[m] = x-pair t + 16 m of this half-warp's plane;
    // false if the TMA form's wait for the slot's copy expired.
    auto inverse_row = [&](int f, V (&r)[16]) -> bool {
        if constexpr (TMA) {
            bool ok = tid != 0 || stage_wait(smem_addr(&stageFull[f % NST]), (f / NST) & 1);
            // Expired-wait test: once slot 0's copy has landed (no copy is then
            // in flight), a short bounded wait on a barrier nothing signals
            // runs out and takes the path of any expired wait.
            if (tid == 0 && ok && f == 0 && a.expireWaitForTest != 0)
                ok = stage_wait(smem_addr(&never), 0, 1LL << 14);
            if (!__syncthreads_and(ok)) {
                if (tid == 0 && a.error != nullptr) atomicExch(a.error, 1);
                return false;
            }
        } else {
            cp_async_wait_all();
            __syncthreads();
        }
        // The stage refilled here was last read in the previous slot, before
        // this barrier.
        if (f + NST - 1 < a.fieldsIn) issue(f + NST - 1);
        const V* st = stage_of(f) + pl * KP;
        const unsigned char* stb = reinterpret_cast<const unsigned char*>(stage_of(f));
        // TMA form: bins k = t + T m and M - k sit at this lane's swizzled
        // offsets plus or minus whole swizzle periods.
        auto bin = [&](int m, bool mirror) -> V {
            if constexpr (TMA) {
                const int rows = (m / PER) * PER * T * B * 8;
                return *reinterpret_cast<const V*>(stb + (mirror ? tmaHi[m % PER] - rows : tmaLo[m % PER] + rows));
            } else {
                return st[mirror ? M - t - T * m : t + T * m];
            }
        };
        // keep <= 11 T (checked at launch): bins k >= 11 T (m >= 11) and
        // M - k > 11 T (m <= 4) lie beyond the 2/3 band and are zero, so those
        // shared-memory reads are left out.
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int k = t + T * m;
            V xk = m < 11 ? bin(m, false) : V{0.f, 0.f};
            V xm = m > 4 ? bin(m, true) : V{0.f, 0.f};
            if (m == 0 && t == 0) {  // bins 0 and M are real
                xk.y = 0.f;
                xm.y = 0.f;
            }
            const V sum = cadd(xk, cconj(xm));
            const V d = csub(xk, cconj(xm));
            const V tt = cmulc(d, tf[k]);
            r[m] = {sum.x - tt.y, sum.y + tt.x};
        }
        __syncwarp();  // the previous transform's reads of the exchange are done
        fft_regs<float, M, 16, +1, 1, false>(r, t, tw2, xch);
        return true;
    };

    grid_wait();
    if constexpr (TMA) __syncthreads();  // barrier init and zero rows before the first copy and reads
    for (int f = 0; f < NST - 1 && f < a.fieldsIn; ++f) issue(f);
    V u[16], v[16], w[16];
    if (!inverse_row(0, u) || !inverse_row(1, v) || !inverse_row(2, w)) return;
    if constexpr (WSM) {
#pragma unroll
        for (int e = 0; e < 16; ++e) wsm[e * NT + tid] = w[e];
    }
    const float scale = a.scale;
    // Lane holding Z[M - k].
    const int src = PAIRED ? 2 * ((T - t) & (T - 1)) + (lane & 1) : ((T - t) & (T - 1)) + (lane & ~(T - 1));
    for (int tg = 0; tg < a.targets; ++tg) {
        V acc[16], q[16];
        if (!inverse_row(3 + 3 * tg, q)) return;
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] = {u[e].x * q[e].x, u[e].y * q[e].y};
        if (!inverse_row(4 + 3 * tg, q)) return;
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] = {acc[e].x + v[e].x * q[e].x, acc[e].y + v[e].y * q[e].y};
        if (!inverse_row(5 + 3 * tg, q)) return;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const V we = WSM ? wsm[e * NT + tid] : w[e];
            acc[e] = {-scale * (acc[e].x + we.x * q[e].x), -scale * (acc[e].y + we.y * q[e].y)};
        }
        __syncwarp();
        fft_regs<float, M, 16, -1, 1, false>(acc, t, tw2, xch);
        // Real-spectrum split, kx < keep, into [k][b].  Z[M - k] for k = t + T k1
        // is register 15 - k1 of lane T - t (t > 0) or register (16 - k1) mod 16
        // of this lane (t = 0).
#pragma unroll
        for (int k1 = 0; k1 < 11; ++k1) {  // k < 11 T >= keep
            const V other = {__shfl_sync(0xFFFFFFFFu, acc[15 - k1].x, src),
                             __shfl_sync(0xFFFFFFFFu, acc[15 - k1].y, src)};
            const int k = t + T * k1;
            const V zk = acc[k1];
            const V zm = cconj(t == 0 ? acc[(16 - k1) & 15] : other);
            V X;
            if (k == 0) {
                X = {zk.x + zk.y, 0.f};
            } else {
                const V ev = cscale(cadd(zk, zm), 0.5f);
                const V d = csub(zk, zm);
                const V o = {0.5f * d.y, -0.5f * d.x};
                X = cadd(ev, cmul(tf[k < M ? k : 0], o));
            }
            if (k < keep) outTile[outSlot(k, pl)] = X;
        }
        __syncthreads();
        if (cok) {
            const long long plane = (static_cast<long long>(member) * a.targets + tg) * a.zStride + z0 + cb;
            V* dst = out + plane + outRow * (a.binsOut.kxStride * y + ck);
            for (int k = ck; k < keep; k += KSTEP, dst += outRow * KSTEP) *dst = outTile[outSlot(k, cb)];
        }
        // The next outTile write happens after the next inverse_row's barrier.
    }
}

template <int M, int B, int MINB, int NS>
cudaError_t launch_pair(const RowFluxArgs& a, cudaStream_t stream) {
    constexpr bool TMA = NS != 0;
    const int zChunks = (a.nz + B - 1) / B;
    const dim3 grid(unsigned(zChunks * a.members), unsigned(a.ny));
    auto kernel = rows_flux_pair_kernel<M, B, MINB, NS>;
    CUtensorMap map{};
    size_t bytes = sizeof(float2) * pair_smem_words<B>(a.keep);
    if constexpr (TMA) {
        // The input bins as [cell][plane]: a cell's planes are contiguous and
        // cells (ky * kxStride + kx) lie `planes` values apart.
        const cudaError_t merr =
            encode_complex_map_2d(&map, a.binsIn.data, static_cast<unsigned long long>(a.binsIn.planes),
                                  static_cast<unsigned long long>(a.ny) * a.binsIn.kxStride,
                                  static_cast<unsigned long long>(a.binsIn.planes) * 8, B, a.keep);
        if (merr != cudaSuccess) return merr;
        bytes = pair_tma_smem_bytes<M, B, NS, pair_w_in_smem<M, B, MINB, NS>()>(a.keep);
    }
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
    if (err != cudaSuccess) return err;
    return launch_chained(kernel, grid, M / 16 * B, bytes, stream, a, map);
}

template <int NS>
cudaError_t launch_pair_form(const RowFluxArgs& a, cudaStream_t stream) {
    constexpr int M = kPairM;
    if (a.planes == 8) return a.pairs == 2 ? launch_pair<M, 8, 3, NS>(a, stream) : launch_pair<M, 8, 2, NS>(a, stream);
    if (a.planes == 16) return launch_pair<M, 16, 1, NS>(a, stream);
    // 24 planes (12 warps, one CTA per SM, 192-byte pieces): cp.async only,
    // no TMA swizzle pattern fits a 192-byte row.
    if (a.planes == 24) return launch_pair<M, 24, 1, 0>(a, stream);
    return cudaErrorInvalidValue;
}

// 256- and 128-point rows: four or eight planes per warp, TMA stages, at the
// same 12 warps per SM.
template <int M>
cudaError_t launch_short_rows(const RowFluxArgs& a, cudaStream_t stream) {
    if (a.planes >= 16) return launch_pair<M, 16, 3 * 256 * 8 / (M * 16), 2>(a, stream);
    return launch_pair<M, 8, 3 * 256 * 8 / (M * 8), 2>(a, stream);
}

}  // namespace

template <int M, int B>
cudaError_t launch_m(const RowFluxArgs& a, cudaStream_t stream) {
    const int zChunks = (a.nz + B - 1) / B;
    const dim3 grid(unsigned(zChunks * a.members), unsigned(a.ny));
    auto kernel = rows_flux_kernel<M, B>;
    const size_t bytes = sizeof(float2) * rows_smem_words<M, B>(a.keep);
    if (bytes > 48 * 1024) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
        if (err != cudaSuccess) return err;
    }
    kernel<<<grid, 32 * B, bytes, stream>>>(a);
    return cudaGetLastError();
}

template <int M>
cudaError_t launch_planes(const RowFluxArgs& a, cudaStream_t stream) {
    switch (a.planes) {
        case 4: return launch_m<M, 4>(a, stream);
        case 8: return launch_m<M, 8>(a, stream);
        case 16: return launch_m<M, 16>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_rows_flux(const RowFluxArgs& a, cudaStream_t stream) {
    const int M = a.nx / 2;
    if (a.keep < 1 || a.keep > M + 1 || a.fieldsIn != 3 + 3 * a.targets || a.zStride < a.nz) return cudaErrorInvalidValue;
    // The TMA forms need the error word (their copy waits are bounded) and
    // 16-byte aligned cells.
    const bool tmaReady = a.error != nullptr && a.binsIn.planes % 2 == 0 && a.zStride % 2 == 0;
    if (M == 128 || M == 64) {
        if (!tmaReady || a.keep > pair_keep(M)) return cudaErrorInvalidValue;
        return M == 128 ? launch_short_rows<128>(a, stream) : launch_short_rows<64>(a, stream);
    }
    if (a.pairs != 0 && M == kPairM && a.keep <= pair_keep(M) && (a.planes == 8 || a.planes == 16 || a.planes == 24)) {
        if (a.tma == 0 || !tmaReady) return launch_pair_form<0>(a, stream);
        return a.tma == 2 ? launch_pair_form<3>(a, stream) : launch_pair_form<2>(a, stream);
    }
    switch (M) {
        case 32: return launch_planes<32>(a, stream);
        case 256: return launch_planes<256>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

bool rows_flux_supported(long long nx) { return nx >= 64 && nx <= 512 && (nx & (nx - 1)) == 0; }

}  // namespace skb
