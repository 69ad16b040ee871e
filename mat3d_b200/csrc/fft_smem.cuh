// fft_smem.cuh -- mixed-radix Stockham FFT stages on lines held in shared memory.
//
// A CTA holds a set of complex lines in shared memory and transforms all of
// them cooperatively: in each stage every thread loops over (line, butterfly)
// work items, reads R inputs from buffer `a`, applies the stage twiddles, does
// an R-point DFT in registers and writes R outputs to buffer `b` (autosort, so
// the result is in natural order without a bit-reversal pass).  Stage s with
// radix R and Ns = product of the previous radices:
//     v[r]  = a[j + r*(n/R)]                    r = 0..R-1, j = 0..n/R-1
//     v[r] *= w_n^( (j mod Ns) * r * n/(Ns*R) )
//     v     = DFT_R(v)
//     b[(j/Ns)*Ns*R + (j mod Ns) + r*Ns] = v[r]
// Twiddles come from a per-length table tw[m] = exp(-2 pi i m / n) in shared
// memory (computed on the host in long double); the inverse uses conj().
// Radices 2 ... 16 of the factors 2, 3 and 5 have dedicated register DFTs, odd
// primes up to 31 (e.g. 13 for n = 65) paired-input butterflies.  Plans take as
// few stages as these radices allow (75 = 15 x 5): every stage costs a shared
// read and write of each point and a barrier.
//
// Line addressing is two-level so one routine serves every pass layout:
//     element e of line L lives at  (L / lpg) * gstride + (L % lpg) * lstride + e * estride
// and `lines_fast` chooses whether consecutive threads walk lines (column
// tiles: consecutive columns are consecutive words, no bank conflicts) or
// butterflies (contiguous lines).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace m3d {

constexpr int kMaxStages = 12;
constexpr int kSMs = 148;  // of a B200: what launch grids and their rules count in

// x / d for 0 <= x, 1 <= d with x * d < 2^32 (always true for indices of a
// shared-memory tile): round-up reciprocal m = ceil(2^32 / d), q = hi32(x m).
// The error of x m / 2^32 against x / d is below x / 2^32 < 1 / d, too small
// to carry the quotient past the next integer.
struct FastDiv {
    unsigned m;
    int d;
    __host__ __device__ __forceinline__ void init(int dd) {
        d = dd;
        m = dd > 1 ? 0xFFFFFFFFu / (unsigned)dd + 1u : 0u;
    }
    __device__ __forceinline__ int div(int x) const { return d == 1 ? x : (int)__umulhi((unsigned)x, m); }
};
inline FastDiv fast_div(int d) {
    FastDiv f;
    f.init(d);
    return f;
}

// per-stage constants shared by every butterfly of a Stockham stage, made on
// the host: a thread runs a handful of butterflies per stage, too few to pay
// for two integer divisions each time
struct StageIdx {
    int R;       // radix
    int step;    // n / (Ns R): twiddle index step
    FastDiv nb;  // n / R: butterflies per line, and the input stride
    FastDiv Ns;  // product of the earlier radices
};

struct LinePlan {
    int n;
    int nstages;
    int radix[kMaxStages];
    StageIdx st[kMaxStages];
    FastDiv dn;  // by n
};
// the derived constants of a plan whose n and radices are set
inline void finish_plan(LinePlan& p) {
    p.dn.init(p.n);
    int Ns = 1;
    for (int s = 0; s < p.nstages; ++s) {
        const int R = p.radix[s];
        p.st[s].R = R;
        p.st[s].nb.init(p.n / R);
        p.st[s].Ns.init(Ns);
        p.st[s].step = p.n / R / Ns;
        Ns *= R;
    }
}

template <typename T> struct Cx;
template <> struct Cx<float> { typedef float2 t; };
template <> struct Cx<double> { typedef double2 t; };

template <typename C2> __device__ __forceinline__ C2 mk(decltype(C2().x) re, decltype(C2().x) im) {
    C2 r; r.x = re; r.y = im; return r;
}
template <typename C2> __device__ __forceinline__ C2 cadd(C2 a, C2 b) { return mk<C2>(a.x + b.x, a.y + b.y); }
template <typename C2> __device__ __forceinline__ C2 csub(C2 a, C2 b) { return mk<C2>(a.x - b.x, a.y - b.y); }
template <typename C2> __device__ __forceinline__ C2 cmul(C2 a, C2 b) {
    return mk<C2>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// multiply by -i (sign < 0) or +i (sign > 0)
template <typename C2> __device__ __forceinline__ C2 crot(C2 a, int sign) {
    return sign < 0 ? mk<C2>(a.y, -a.x) : mk<C2>(-a.y, a.x);
}
template <typename C2> __device__ __forceinline__ C2 twid(const C2* tw, int m, int sign) {
    C2 w = tw[m];
    if (sign > 0) w.y = -w.y;
    return w;
}

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

template <typename C2, int R>
__device__ __forceinline__ void dft_small(C2 (&v)[R], const C2* tw, int n, int sign) {
    typedef decltype(C2().x) T;
    if constexpr (R == 2) {
        C2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4) {
        C2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
        C2 b0 = cadd(v[1], v[3]), b1 = crot(csub(v[1], v[3]), sign);
        v[0] = cadd(a0, b0);
        v[1] = cadd(a1, b1);
        v[2] = csub(a0, b0);
        v[3] = csub(a1, b1);
    } else if constexpr (R == 8) {
        const T h = (T)0.70710678118654752440084436210484903928483593768847L;
        // radix-2 across halves, then two radix-4 on even/odd outputs
        C2 e[4], o[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            e[r] = cadd(v[r], v[r + 4]);
            o[r] = csub(v[r], v[r + 4]);
        }
        // o[r] *= w^r with w = exp(sign * i pi / 4) = (h, sg*h)
        const T sg = (T)sign;
        {
            const T x = o[1].x, y = o[1].y;
            o[1] = mk<C2>(h * (x - sg * y), h * (y + sg * x));
        }
        o[2] = crot(o[2], sign);
        {
            // w^3 = (-h, sg*h)
            const T x = o[3].x, y = o[3].y;
            o[3] = mk<C2>(h * (-x - sg * y), h * (sg * x - y));
        }
        // radix-4 on e -> outputs 0,2,4,6 ; on o -> outputs 1,3,5,7
        C2 a0 = cadd(e[0], e[2]), a1 = csub(e[0], e[2]);
        C2 b0 = cadd(e[1], e[3]), b1 = crot(csub(e[1], e[3]), sign);
        C2 c0 = cadd(o[0], o[2]), c1 = csub(o[0], o[2]);
        C2 d0 = cadd(o[1], o[3]), d1 = crot(csub(o[1], o[3]), sign);
        v[0] = cadd(a0, b0);
        v[4] = csub(a0, b0);
        v[2] = cadd(a1, b1);
        v[6] = csub(a1, b1);
        v[1] = cadd(c0, d0);
        v[5] = csub(c0, d0);
        v[3] = cadd(c1, d1);
        v[7] = csub(c1, d1);
    } else if constexpr (R == 3) {
        const T c = (T)-0.5L;
        const T s = (T)0.86602540378443864676372317075293618347140262690519L * (T)(sign < 0 ? -1 : 1);
        C2 a = v[0], b = v[1], d = v[2];
        C2 t1 = cadd(b, d);
        C2 t2 = mk<C2>(a.x + c * t1.x, a.y + c * t1.y);
        C2 t3 = csub(b, d);  // times i*s
        C2 t3r = mk<C2>(-s * t3.y, s * t3.x);
        v[0] = cadd(a, t1);
        v[1] = cadd(t2, t3r);
        v[2] = csub(t2, t3r);
    } else if constexpr (R == 5) {
        // cos and sin of 72 and 144 degrees
        const T c1 = (T)0.309016994374947424102293417182819L, c2 = (T)-0.809016994374947424102293417182819L;
        const T sg = (T)(sign < 0 ? -1 : 1);
        const T s1 = (T)0.951056516295153572116439333379382L * sg, s2 = (T)0.587785252292473129168705954639073L * sg;
        const C2 a1 = cadd(v[1], v[4]), a2 = cadd(v[2], v[3]), b1 = csub(v[1], v[4]), b2 = csub(v[2], v[3]);
        const C2 t1 = mk<C2>(v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y);
        const C2 t2 = mk<C2>(v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y);
        const C2 u1 = mk<C2>(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y);
        const C2 u2 = mk<C2>(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y);
        v[0] = cadd(v[0], cadd(a1, a2));
        v[1] = mk<C2>(t1.x - u1.y, t1.y + u1.x);
        v[4] = mk<C2>(t1.x + u1.y, t1.y - u1.x);
        v[2] = mk<C2>(t2.x - u2.y, t2.y + u2.x);
        v[3] = mk<C2>(t2.x + u2.y, t2.y - u2.x);
    } else if constexpr (R == 9 || R == 16) {
        // R = P x P: w_R twiddles between two rounds of P-point DFTs
        constexpr int P = R == 9 ? 3 : 4;
        C2 sub[P][P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int m = 0; m < P; ++m) sub[p][m] = v[P * m + p];
            dft_small<C2, P>(sub[p], tw, n, sign);
        }
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
            C2 t[P];
#pragma unroll
            for (int p = 0; p < P; ++p) {
                if (p == 0 || k1 == 0) {
                    t[p] = sub[p][k1];
                } else if constexpr (R == 16) {
                    t[p] = rot_const<C2, 16>(sub[p][k1], p * k1, sign);
                } else {  // cos and sin of 40, 80 and 160 degrees
                    const T c = p * k1 == 1 ? (T)0.766044443118978035202392650555417L
                                            : (p * k1 == 2 ? (T)0.173648177666930348851716626769315L
                                                           : (T)-0.939692620785908384054109277324731L);
                    const T sn = p * k1 == 1 ? (T)0.642787609686539326322643409907263L
                                             : (p * k1 == 2 ? (T)0.984807753012208059366743024589523L
                                                            : (T)0.342020143325668733044099614682260L);
                    t[p] = cmul(sub[p][k1], mk<C2>(c, sign < 0 ? -sn : sn));
                }
            }
            dft_small<C2, P>(t, tw, n, sign);
#pragma unroll
            for (int k2 = 0; k2 < P; ++k2) v[k1 + P * k2] = t[k2];
        }
    } else if constexpr (R == 6 || R == 10 || R == 12 || R == 15) {
        // R = P x Q, coprime: no twiddles between (Good's index maps)
        constexpr int P = R == 12 ? 4 : (R == 15 ? 3 : 2), Q = R / P;
        C2 sub[P][Q];
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int q = 0; q < Q; ++q) sub[p][q] = v[(Q * p + P * q) % R];
            dft_small<C2, Q>(sub[p], tw, n, sign);
        }
        // output k with k mod P = p, k mod Q = q: k = (p ep + q eq) mod R
        constexpr int ep = R == 6 ? 3 : (R == 10 ? 5 : (R == 12 ? 9 : 10)), eq = R == 6 ? 4 : (R == 10 ? 6 : (R == 12 ? 4 : 6));
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            C2 t[P];
#pragma unroll
            for (int p = 0; p < P; ++p) t[p] = sub[p][q];
            dft_small<C2, P>(t, tw, n, sign);
#pragma unroll
            for (int p = 0; p < P; ++p) v[(p * ep + q * eq) % R] = t[p];
        }
    } else {
        // direct DFT through the table: w_R^m = tw[m * (n/R)]
        C2 in[R];
#pragma unroll
        for (int q = 0; q < R; ++q) in[q] = v[q];
        const int st = n / R;
#pragma unroll
        for (int s = 0; s < R; ++s) {
            C2 acc = in[0];
#pragma unroll
            for (int q = 1; q < R; ++q) acc = cadd(acc, cmul(in[q], twid(tw, ((q * s) % R) * st, sign)));
            v[s] = acc;
        }
    }
}

// 9-point DFT as paired sums, inputs m and 9 - m together (see butterfly_odd): about
// the operations of the two rounds of 3-point DFTs of dft_small, and a single
// transform of 27, 81, 171 or 729 points is 4, 10, 9 or 19% nearer its exact values
// with it.  The reconstruction, which offers plain transforms, takes it.  The solvers
// do not: their forward and inverse transforms undo each other's rounding better with
// the 3-point rounds (FP64 strains of thermal 27^3 and 81^3 12 and 17% nearer the
// 64-bit results, of plane 81^2, 243^2 and 486^2 24, 23 and 22%).
template <typename C2>
__device__ __forceinline__ void dft9_paired(C2 (&v)[9], int sign) {
    typedef decltype(C2().x) T;
    const T cs[9] = {(T)1, (T)0.766044443118978035202392650555417L, (T)0.173648177666930348851716626769315L, (T)-0.5,
                     (T)-0.939692620785908384054109277324731L, (T)-0.939692620785908384054109277324731L, (T)-0.5,
                     (T)0.173648177666930348851716626769315L, (T)0.766044443118978035202392650555417L};
    const T sn[9] = {(T)0, (T)0.642787609686539326322643409907263L, (T)0.984807753012208059366743024589523L,
                     (T)0.866025403784438646763723170752936L, (T)0.342020143325668733044099614682260L,
                     (T)-0.342020143325668733044099614682260L, (T)-0.866025403784438646763723170752936L,
                     (T)-0.984807753012208059366743024589523L, (T)-0.642787609686539326322643409907263L};
    C2 a[4], b[4], out[8];
    C2 sum = v[0];
#pragma unroll
    for (int m = 1; m < 5; ++m) {
        a[m - 1] = cadd(v[m], v[9 - m]);
        b[m - 1] = csub(v[m], v[9 - m]);
        sum = cadd(sum, a[m - 1]);
    }
#pragma unroll
    for (int k = 1; k < 5; ++k) {
        C2 A = v[0], B = mk<C2>(0, 0);
#pragma unroll
        for (int m = 1; m < 5; ++m) {
            const T c = cs[k * m % 9], d = sign < 0 ? -sn[k * m % 9] : sn[k * m % 9];
            A.x += c * a[m - 1].x;
            A.y += c * a[m - 1].y;
            B.x += d * b[m - 1].x;
            B.y += d * b[m - 1].y;
        }
        out[k - 1] = mk<C2>(A.x - B.y, A.y + B.x);
        out[8 - k] = mk<C2>(A.x + B.y, A.y - B.x);
    }
    v[0] = sum;
#pragma unroll
    for (int k = 1; k < 9; ++k) v[k] = out[k - 1];
}

// butterfly j of a stage: inputs j + r nb, twiddles w^(k r step) with
// j = g Ns + k, outputs g Ns R + k + r Ns
template <typename C2, int R, bool Paired9 = false>
__device__ __forceinline__ void butterfly(const C2* __restrict__ src, C2* __restrict__ dst, int j, int g, int k,
                                          const StageIdx& S, int es, const C2* tw, int sign) {
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[(j + r * S.nb.d) * es];
    if (S.Ns.d > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul(v[r], twid(tw, k * r * S.step, sign));
    }
    if constexpr (R == 9 && Paired9) dft9_paired(v, sign);
    else dft_small<C2, R>(v, tw, S.nb.d * R, sign);
    const int idx = g * S.Ns.d * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[(idx + r * S.Ns.d) * es] = v[r];
}

// Odd prime radix R >= 7, compile time: inputs j and R-j are paired
// (a_j = x_j + x_{R-j}, b_j = x_j - x_{R-j}) so outputs k and R-k share one set
// of products:
//   y_k, y_{R-k} = x_0 + sum_j a_j cos(2 pi jk/R) +- i sign sum_j b_j sin(2 pi jk/R)
// -- (R-1)^2 real multiply-adds per butterfly instead of the 4 R^2 of a direct
// DFT.  Outputs go straight to `dst`, so only a, b and the h = (R-1)/2 cosines
// and sines (from the table: tw[m n/R] = (cos, -sin) of 2 pi m/R) live in
// registers.
template <typename C2, int R>
__device__ __forceinline__ void butterfly_odd(const C2* __restrict__ src, C2* __restrict__ dst, int j, int g, int k0,
                                              const StageIdx& S, int es, const C2* tw, int sign) {
    typedef decltype(C2().x) T;
    constexpr int h = (R - 1) / 2;
    const int nb = S.nb.d, Ns = S.Ns.d, step = S.step;
    const C2 x0 = src[j * es];
    C2 a[h], b[h];
#pragma unroll
    for (int q = 1; q <= h; ++q) {
        C2 u = src[(j + q * nb) * es], w = src[(j + (R - q) * nb) * es];
        if (Ns > 1) {
            u = cmul(u, twid(tw, k0 * q * step, sign));
            w = cmul(w, twid(tw, k0 * (R - q) * step, sign));
        }
        a[q - 1] = cadd(u, w);
        b[q - 1] = csub(u, w);
    }
    T c[h], sn[h];
#pragma unroll
    for (int m = 1; m <= h; ++m) {
        const C2 w = tw[m * nb];
        c[m - 1] = w.x;
        sn[m - 1] = sign < 0 ? w.y : -w.y;  // sign * sin(2 pi m / R)
    }
    const int idx = g * Ns * R + k0;
    C2 y0 = x0;
#pragma unroll
    for (int q = 0; q < h; ++q) y0 = cadd(y0, a[q]);
    dst[idx * es] = y0;
#pragma unroll
    for (int k = 1; k <= h; ++k) {
        T px = x0.x, py = x0.y, qx = 0, qy = 0;
#pragma unroll
        for (int q = 1; q <= h; ++q) {
            const int m = (q * k) % R;  // never 0: R is prime
            const T cc = m <= h ? c[m - 1] : c[R - m - 1];
            const T ss = m <= h ? sn[m - 1] : -sn[R - m - 1];
            px += a[q - 1].x * cc;
            py += a[q - 1].y * cc;
            qx += b[q - 1].x * ss;
            qy += b[q - 1].y * ss;
        }
        dst[(idx + k * Ns) * es] = mk<C2>(px - qy, py + qx);
        dst[(idx + (R - k) * Ns) * es] = mk<C2>(px + qy, py - qx);
    }
}

// generic-radix butterfly (any R up to kMaxGenericRadix), run-time R
constexpr int kMaxGenericRadix = 32;
template <typename C2>
__device__ __noinline__ void butterfly_generic(const C2* __restrict__ src, C2* __restrict__ dst, int R, int j, int g,
                                               int k, const StageIdx& S, int es, const C2* tw, int sign) {
    typedef decltype(C2().x) T;
    const int nb = S.nb.d, Ns = S.Ns.d, step = S.step;
    C2 v[kMaxGenericRadix];
    for (int r = 0; r < R; ++r) v[r] = src[(j + r * nb) * es];
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], twid(tw, k * r * step, sign));
    const int st = nb;
    const int idx = g * Ns * R + k;
    for (int s = 0; s < R; ++s) {
        C2 acc = v[0];
        for (int q = 1; q < R; ++q) acc = cadd(acc, cmul(v[q], twid(tw, ((q * s) % R) * st, sign)));
        dst[(idx + s * Ns) * es] = acc;
    }
    (void)sizeof(T);
}

struct LineLayout {
    int nlines;   // number of lines
    int lpg;      // lines per group
    int lstride;  // stride between lines inside a group
    int gstride;  // stride between groups
    int estride;  // stride between elements of a line
    bool lines_fast;
};

// Transforms every line; returns the buffer (a or b) that holds the result.
// Must be called by all threads of the CTA; ends with __syncthreads().
// Radices 2 ... 16 of the factors 2, 3 and 5 are compile-time butterflies; the
// odd primes 7..MaxR are compile-time too when MaxR reaches them (each adds
// registers to the kernel, so callers pick the smallest MaxR their lengths
// need); any other radix runs the run-time generic butterfly.
// one Stockham stage of radix R over every line of the tile (R fixed at
// compile time, so the loop body is one straight-line butterfly); KIND 0 =
// butterfly (radices of 2, 3 and 5 up to 16), 1 = butterfly_odd (primes from 7), 2 =
// run-time generic, 3 = butterfly with the paired 9-point DFT
template <typename C2, int R, int KIND>
__device__ __forceinline__ void run_stage(const C2* a, C2* b, const C2* tw, const StageIdx& S, int Rrt,
                                          const LineLayout& L, const FastDiv& dl, const FastDiv& dg, int sign) {
    const int total = S.nb.d * L.nlines;
    const int es = L.estride;
    for (int w = threadIdx.x; w < total; w += blockDim.x) {
        int line, j;
        if (L.lines_fast) { j = dl.div(w); line = w - j * L.nlines; }
        else { line = S.nb.div(w); j = w - line * S.nb.d; }
        const int grp = dg.div(line);
        const int base = grp * L.gstride + (line - grp * L.lpg) * L.lstride;
        const int g = S.Ns.div(j), k = j - g * S.Ns.d;
        if constexpr (KIND == 0 || KIND == 3) butterfly<C2, R, KIND == 3>(a + base, b + base, j, g, k, S, es, tw, sign);
        else if constexpr (KIND == 1) butterfly_odd<C2, R>(a + base, b + base, j, g, k, S, es, tw, sign);
        else butterfly_generic<C2>(a + base, b + base, Rrt, j, g, k, S, es, tw, sign);
    }
}

template <typename C2, int MaxR = 5, bool Paired9 = false>
__device__ __forceinline__ C2* fft_lines(C2* a, C2* b, const C2* tw, const LinePlan& p, const LineLayout& L, int sign) {
    FastDiv dl, dg;  // by the lines of the tile, by the lines of a group
    dl.init(L.nlines);
    dg.init(L.lpg);
    for (int s = 0; s < p.nstages; ++s) {
        const StageIdx& S = p.st[s];
        const int R = S.R;
        switch (R) {
            case 2: run_stage<C2, 2, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 3: run_stage<C2, 3, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 4: run_stage<C2, 4, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 5: run_stage<C2, 5, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 6: run_stage<C2, 6, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 8: run_stage<C2, 8, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 9: run_stage<C2, 9, Paired9 ? 3 : 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 10: run_stage<C2, 10, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 12: run_stage<C2, 12, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 15: run_stage<C2, 15, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            case 16: run_stage<C2, 16, 0>(a, b, tw, S, R, L, dl, dg, sign); break;
            default:
                if constexpr (MaxR >= 7) if (R == 7) { run_stage<C2, 7, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 11) if (R == 11) { run_stage<C2, 11, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 13) if (R == 13) { run_stage<C2, 13, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 17) if (R == 17) { run_stage<C2, 17, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 19) if (R == 19) { run_stage<C2, 19, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 23) if (R == 23) { run_stage<C2, 23, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 29) if (R == 29) { run_stage<C2, 29, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                if constexpr (MaxR >= 31) if (R == 31) { run_stage<C2, 31, 1>(a, b, tw, S, R, L, dl, dg, sign); break; }
                run_stage<C2, 1, 2>(a, b, tw, S, R, L, dl, dg, sign);
                break;
        }
        __syncthreads();
        C2* t = a; a = b; b = t;
    }
    return a;
}

}  // namespace m3d
