// fft_reg.cuh -- compile-time-sized FFT of one line spread over T lanes of a warp.
//
// A line of N = E*T points is transformed by the four-step split
//     X[k1 + E k2] = sum_t w_T^(t k2) w_N^(t k1) sum_j w_E^(j k1) x[t + T j]
// Lane t of the line holds E points in registers:
//   natural distribution : v[j]          = x[t + T j],            j < E
//   spectral distribution: v[q*T + k2]   = X[(t*Q + q) + E k2],   q < Q = E/T, k2 < T
// line_fwd maps natural -> spectral: a radix-E DFT in registers, the w_N
// twiddles, one exchange through shared memory among the T lanes of the line
// (warp-synchronous, no block barrier), and Q radix-T DFTs in registers.
// line_inv is the transposed algorithm and maps spectral -> natural, so a
// forward + pointwise + inverse sequence needs no reordering at all.
// The in-register DFTs are mixed-radix (2, 3, 4, 5, 8) decimation in time
// with every index a compile-time constant; twiddles are read from the
// per-line table tw[m] = exp(-2 pi i m / N) held in shared memory.
#pragma once
#include "fft_smem.cuh"

namespace m3d {

// exp(-+2 pi i m / L) for L dividing 96, m known at compile time: the sub-DFT
// twiddles inside the register DFTs.  As immediates they cost neither the
// broadcast shared-memory loads nor the registers of table entries (a radix-24
// DFT multiplies by 15 of them); thermal 128^3 refinement 11.44 -> 11.33 ms a
// solve.  Not for the radix-32 DFT, whose y forward pass at FP32 256^3 went from
// 102 to 155 us with them.  cos and sin of
// 2 pi k / 96 in the first octant, mirrored into the others; the switches fold
// away once the loops over m are unrolled.
template <typename T>
__device__ __forceinline__ void octant96(int k, T& c, T& s) {
    switch (k) {
        case 0: c = (T)1.0000000000000000000000; s = (T)0.0; break;
        case 1: c = (T)0.9978589232386035067380; s = (T)0.0654031292301430668153; break;
        case 2: c = (T)0.9914448613738104111445; s = (T)0.1305261922200515915484; break;
        case 3: c = (T)0.9807852804032304491261; s = (T)0.1950903220161282678482; break;
        case 4: c = (T)0.9659258262890682867497; s = (T)0.2588190451025207623488; break;
        case 5: c = (T)0.9469301294951056642558; s = (T)0.3214394653031615807010; break;
        case 6: c = (T)0.9238795325112867561281; s = (T)0.3826834323650897717284; break;
        case 7: c = (T)0.8968727415326883038941; s = (T)0.4422886902190012819952; break;
        case 8: c = (T)0.8660254037844386467637; s = (T)0.5000000000000000000000; break;
        case 9: c = (T)0.8314696123025452370787; s = (T)0.5555702330196022247428; break;
        case 10: c = (T)0.7933533402912351645797; s = (T)0.6087614290087206394160; break;
        case 11: c = (T)0.7518398074789773964075; s = (T)0.6593458151000688684251; break;
        default: c = (T)0.7071067811865475244008; s = (T)0.7071067811865475244008; break;
    }
}
// a * exp(sign 2 pi i m / L)
template <typename C2, int L>
__device__ __forceinline__ C2 rot_const(C2 a, int m, int sign) {
    typedef decltype(C2().x) T;
    static_assert(96 % L == 0, "twiddles of a divisor of 96 points");
    m = (m * (96 / L)) % 96;
    const int quad = m / 24, r = m % 24;  // angle = quad * 90 degrees + r
    T c, s;
    if (r > 12) octant96<T>(24 - r, s, c);
    else octant96<T>(r, c, s);
    const T cv = quad == 0 ? c : (quad == 1 ? -s : (quad == 2 ? -c : s));
    const T sv = quad == 0 ? s : (quad == 1 ? c : (quad == 2 ? -s : -c));
    return cmul(a, mk<C2>(cv, sign < 0 ? -sv : sv));
}

// DFT of compile-time length L in registers; tw: the table of NL points
// (w_L^m = tw[m * (NL/L)]) for radices 5 and 32.
template <typename C2, int L, int NL>
__device__ __forceinline__ void dft_reg(C2 (&v)[L], const C2* tw, int sign) {
    static_assert(NL % L == 0, "sub-DFT length must divide the table length");
    if constexpr (L == 1) {
        return;
    } else if constexpr (L == 2 || L == 3 || L == 4 || L == 5 || L == 8) {
        dft_small<C2, L>(v, tw, NL, sign);
    } else {
        constexpr int P = (L % 4 == 0) ? 4 : ((L % 2 == 0) ? 2 : ((L % 3 == 0) ? 3 : 5));
        constexpr int Q = L / P;
        C2 sub[P][Q];
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int m = 0; m < Q; ++m) sub[p][m] = v[P * m + p];
#pragma unroll
        for (int p = 0; p < P; ++p) dft_reg<C2, Q, NL>(sub[p], tw, sign);
#pragma unroll
        for (int p = 1; p < P; ++p)
#pragma unroll
            for (int k1 = 1; k1 < Q; ++k1) sub[p][k1] = L < 32 ? rot_const<C2, L>(sub[p][k1], p * k1, sign)
                                    : cmul(sub[p][k1], twid(tw, p * k1 * (NL / L), sign));
#pragma unroll
        for (int k1 = 0; k1 < Q; ++k1) {
            C2 t[P];
#pragma unroll
            for (int p = 0; p < P; ++p) t[p] = sub[p][k1];
            dft_small<C2, P>(t, tw, NL, sign);
#pragma unroll
            for (int k2 = 0; k2 < P; ++k2) v[k1 + Q * k2] = t[k2];
        }
    }
}

// Line split for each supported length and element type: N = E * T, T | E,
// T lanes per line (so 32/T lines per warp).
template <typename T, int N> struct LineSplit;
#define M3D_SPLIT(TY, NN, EE, TT) \
    template <> struct LineSplit<TY, NN> { static constexpr int E = EE, Tl = TT; };
M3D_SPLIT(float, 16, 4, 4)
M3D_SPLIT(float, 32, 8, 4)
M3D_SPLIT(float, 48, 12, 4)
M3D_SPLIT(float, 64, 8, 8)
M3D_SPLIT(float, 96, 24, 4)
M3D_SPLIT(float, 128, 16, 8)
M3D_SPLIT(float, 256, 32, 8)
M3D_SPLIT(double, 16, 4, 4)
M3D_SPLIT(double, 32, 8, 4)
M3D_SPLIT(double, 48, 12, 4)
M3D_SPLIT(double, 64, 8, 8)
M3D_SPLIT(double, 96, 24, 4)
M3D_SPLIT(double, 128, 16, 8)
M3D_SPLIT(double, 256, 16, 16)
#undef M3D_SPLIT

constexpr bool fast_size(int n) {
    return n == 16 || n == 32 || n == 48 || n == 64 || n == 96 || n == 128 || n == 256;
}

// exchange buffer of one line: element (k1, t) at k1*(T+1) + t
template <int E, int T> struct Xch { static constexpr int size = E * (T + 1) + 1; };

// Exchange element (k1, t) lives at k1*(T+1) + (t ^ sw); `sw` (0 or 1) is a
// per-line bank swizzle chosen with the row padding (BankCfg in
// passes_fast.cuh) so that the natural, spectral and both exchange access
// patterns of a warp are conflict-free.
template <typename C2, int E, int T>
__device__ __forceinline__ void line_fwd(C2 (&v)[E], int t, C2* xch, const C2* tw, int sw = 0) {
    constexpr int N = E * T, Q = E / T;
    dft_reg<C2, E, N>(v, tw, -1);
#pragma unroll
    for (int k1 = 1; k1 < E; ++k1) v[k1] = cmul(v[k1], twid(tw, t * k1, -1));
    const int ts = t ^ sw;
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) xch[k1 * (T + 1) + ts] = v[k1];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        C2 u[T];
#pragma unroll
        for (int t2 = 0; t2 < T; ++t2) u[t2] = xch[(t * Q + q) * (T + 1) + (t2 ^ sw)];
        dft_reg<C2, T, N>(u, tw, -1);
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) v[q * T + k2] = u[k2];
    }
    __syncwarp();
}

template <typename C2, int E, int T>
__device__ __forceinline__ void line_inv(C2 (&v)[E], int t, C2* xch, const C2* tw, int sw = 0) {
    constexpr int N = E * T, Q = E / T;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        C2 u[T];
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) u[k2] = v[q * T + k2];
        dft_reg<C2, T, N>(u, tw, +1);
        const int k1 = t * Q + q;
#pragma unroll
        for (int t2 = 0; t2 < T; ++t2) {
            const C2 w = (t2 == 0) ? u[t2] : cmul(u[t2], twid(tw, t2 * k1, +1));
            xch[k1 * (T + 1) + (t2 ^ sw)] = w;
        }
    }
    __syncwarp();
    const int ts = t ^ sw;
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) v[k1] = xch[k1 * (T + 1) + ts];
    __syncwarp();
    dft_reg<C2, E, N>(v, tw, +1);
}

// mode index held in v[r] (spectral distribution) by lane t
template <int E, int T>
__device__ __forceinline__ int spec_mode(int t, int r) {
    constexpr int Q = E / T;
    return (t * Q + r / T) + E * (r % T);
}

}  // namespace m3d
