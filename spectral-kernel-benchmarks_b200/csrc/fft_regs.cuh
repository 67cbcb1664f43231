// Register-ended batched FFT of the horizontal transform kernels.
//
// A length-N sequence is owned by T = N / E threads; thread t holds elements
// t + T e (e < E) in v[e], before and after the transform.  Passes are Stockham
// auto-sort passes of radix E (the last one of the radix that remains): pass
// with current sub-transform size Ns and radix R reads butterfly j's inputs
// j + r N/R, which for j = t + T s (s < E/R) are the thread's own registers
// s + r E/R, so a pass touches no memory; between passes the values go through
// an exchange buffer to their Stockham positions (j/Ns) Ns R + j mod Ns + r Ns
// and come back as elements t + T e.  With E = 16 a 128- or 256-point transform
// is two radix-16 / radix-8 passes and one exchange, 512 points are three
// passes and two exchanges.
//
// Why registers: the transform kernels are bound by the L1 / shared-memory
// pipe, not by arithmetic (FP64 256-point columns with three radix-8/4 passes
// through shared memory ran that pipe at 83 %, DRAM at 36 %): staging the
// loads, two accesses per pass and a read-back were eight shared accesses per
// element, where one exchange is two.
//
// Twiddles exp(-2 pi i k / N) (host-generated in long double; the inverse
// direction uses the conjugates) come from a table in the order the threads
// read it (regs_table_index): pass by pass, [r - 1][j mod Ns], so that threads
// with consecutive t read consecutive entries.  Read from the natural table,
// entry (j mod Ns) r N / (Ns R), the lanes of a row kernel's warp touched up to
// eight cache lines per load.

#pragma once

#include "fft_device.cuh"

namespace skb {

// W16^e with exponent sign SIGN, e in {1, 2, 3, 6, 9} (e = 4 is a
// multiplication by SIGN*i): cos(2 pi e / 16) + SIGN i sin(2 pi e / 16).
template <int SIGN, int E, typename V>
__device__ __forceinline__ V w16() {
    using S = decltype(V{}.x);
    constexpr S c1 = S(0.923879532511286756128183189396788286822L);  // cos(pi/8)
    constexpr S s1 = S(0.382683432365089771728459984030398866761L);  // sin(pi/8)
    constexpr S h = S(0.707106781186547524400844362104849039285L);   // cos(pi/4)
    constexpr S sg = SIGN < 0 ? S(-1) : S(1);
    if constexpr (E == 1) return {c1, sg * s1};
    if constexpr (E == 2) return {h, sg * h};
    if constexpr (E == 3) return {s1, sg * c1};
    if constexpr (E == 6) return {-h, sg * h};
    return {-c1, -sg * s1};  // E == 9
}

// In-place length-16 DFT over v[0..15] (natural order in and out): 16 = 4 x 4,
// input m = m2 + 4 m1, output k = k1 + 4 k2.
template <int SIGN, typename V>
__device__ __forceinline__ void dft16(V* v) {
#pragma unroll
    for (int m2 = 0; m2 < 4; ++m2) dft4<SIGN>(v[m2], v[m2 + 4], v[m2 + 8], v[m2 + 12]);
    // v[m2 + 4 k1] *= W16^(m2 k1)
    v[5] = cmul(v[5], w16<SIGN, 1, V>());
    v[9] = cmul(v[9], w16<SIGN, 2, V>());
    v[13] = cmul(v[13], w16<SIGN, 3, V>());
    v[6] = cmul(v[6], w16<SIGN, 2, V>());
    v[10] = cmul_si<SIGN>(v[10]);
    v[14] = cmul(v[14], w16<SIGN, 6, V>());
    v[7] = cmul(v[7], w16<SIGN, 3, V>());
    v[11] = cmul(v[11], w16<SIGN, 6, V>());
    v[15] = cmul(v[15], w16<SIGN, 9, V>());
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4<SIGN>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // v[4 k1 + k2] holds output k1 + 4 k2: transpose the 4 x 4 block.
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i + 1; j < 4; ++j) {
            const V t = v[4 * i + j];
            v[4 * i + j] = v[4 * j + i];
            v[4 * j + i] = t;
        }
}

// In-place length-R DFT, natural order in and out.
template <int SIGN, int R, typename V>
__device__ __forceinline__ void dft_small(V* v) {
    static_assert(R == 1 || R == 2 || R == 4 || R == 8 || R == 16, "radix");
    if constexpr (R == 2) dft2<SIGN>(v[0], v[1]);
    if constexpr (R == 4) dft4<SIGN>(v[0], v[1], v[2], v[3]);
    if constexpr (R == 8) dft8<SIGN>(v);
    if constexpr (R == 16) dft16<SIGN>(v);
}

// Exchange among threads (plane b of B, t) with b fastest, [position][plane]:
// runs of B consecutive values, free of bank conflicts when B values fill an
// access phase (128 bytes).
template <typename V, int B>
struct PlaneExchange {
    V* x;  // this thread's plane
    __device__ __forceinline__ void store(int i, V v) { x[i * B] = v; }
    __device__ __forceinline__ V load(int i) const { return x[i * B]; }
    __device__ __forceinline__ void fence() const { __syncthreads(); }
};

// One pass (sub-transforms of Ns points, radix R) on the thread's registers.
// LDG: the table lies in global memory (read through __ldg), else anywhere.
template <typename S, int N, int E, int SIGN, int Ns, bool LDG = true>
__device__ __forceinline__ void fft_regs_pass(cx<S> (&v)[E], int t, const cx<S>* tw) {
    using V = cx<S>;
    constexpr int T = N / E;
    constexpr int R = N / Ns < E ? N / Ns : E;
    constexpr int BF = E / R;  // butterflies of this pass per thread
    static_assert(T * E == N && R * BF == E, "power-of-two lengths");
#pragma unroll
    for (int s = 0; s < BF; ++s) {
        V b[R];
#pragma unroll
        for (int r = 0; r < R; ++r) b[r] = v[s + r * BF];
        if constexpr (Ns > 1) {
            const V* w = tw + (t + T * s) % Ns;
#pragma unroll
            for (int r = 1; r < R; ++r)
                b[r] = cmul(b[r], LDG ? twiddle<SIGN>(w, Ns * (r - 1)) : twiddle_plain<SIGN>(w, Ns * (r - 1)));
        }
        dft_small<SIGN, R>(b);
#pragma unroll
        for (int r = 0; r < R; ++r) v[s + r * BF] = b[r];
    }
}

// Store the pass's results at their Stockham positions.
template <typename S, int N, int E, int Ns, typename X>
__device__ __forceinline__ void fft_regs_store(const cx<S> (&v)[E], int t, X& xch) {
    constexpr int T = N / E;
    constexpr int R = N / Ns < E ? N / Ns : E;
    constexpr int BF = E / R;
#pragma unroll
    for (int s = 0; s < BF; ++s) {
        const int j = t + T * s;
        const int base = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
        for (int r = 0; r < R; ++r) xch.store(base + r * Ns, v[s + r * BF]);
    }
}

// The passes from sub-transform size Ns on; tw points at pass Ns's entries.
// `xch` gives store(position, value), load(position) and fence(), a barrier
// of (at least) the T threads that share the sequence.  For Ns = 1 the exchange
// buffer must be free on entry; loads of the last exchange may still be in
// flight in other threads on return.
template <typename S, int N, int E, int SIGN, int Ns = 1, bool LDG = true, typename X>
__device__ __forceinline__ void fft_regs(cx<S> (&v)[E], int t, const cx<S>* tw, X& xch) {
    constexpr int R = N / Ns < E ? N / Ns : E;
    fft_regs_pass<S, N, E, SIGN, Ns, LDG>(v, t, tw);
    if constexpr (Ns * R < N) {
        if constexpr (Ns > 1) xch.fence();  // the previous exchange's loads
        fft_regs_store<S, N, E, Ns>(v, t, xch);
        xch.fence();
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = xch.load(t + (N / E) * e);
        fft_regs<S, N, E, SIGN, Ns * R, LDG>(v, t, Ns > 1 ? tw + Ns * (R - 1) : tw, xch);
    }
}

// The passes up to sub-transform size `End`, whose results are left in the
// exchange buffer at their positions (a barrier has to follow).
template <typename S, int N, int E, int SIGN, int End, int Ns = 1, typename X>
__device__ __forceinline__ void fft_regs_head(cx<S> (&v)[E], int t, const cx<S>* tw, X& xch) {
    fft_regs_pass<S, N, E, SIGN, Ns>(v, t, tw);
    if constexpr (Ns > 1) xch.fence();
    fft_regs_store<S, N, E, Ns>(v, t, xch);
    if constexpr (Ns * E < End) {
        xch.fence();
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = xch.load(t + (N / E) * e);
        fft_regs_head<S, N, E, SIGN, End, Ns * E>(v, t, Ns > 1 ? tw + Ns * (E - 1) : tw, xch);
    }
}

}  // namespace skb
