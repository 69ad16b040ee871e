// mid_ops.cuh -- the pointwise middle of a sweep, between the z inverse and the
// next z forward, as operators of the fused z kernels (passes_plane.cuh,
// passes_zmid.cuh): In/load the inputs of an item of W consecutive voxels, apply
// the update and return what the forward transform takes.
#pragma once
#include "inelastic.cuh"
#include "physics.cuh"

namespace m3d {

// EM update and polarization of isotropic phases: A d = a_l tr(d) I + a_s d
// and P x likewise, two constants per phase and table instead of 36 (every
// phase of the mechanical solver is isotropic, so C, S, C - C0, S - S0 and
// 2 (C + C0)^-1 C0 are); thermal tables (C = 3) are a_s I and p_s I.
// Sums: [0] sum w d^2.
template <typename T>
struct MidEMArgs {
    const uint8_t* phase;
    T* x;
    const float* r;       // defect forcing of the correction solve, may be null
    long long V;
    const double* P;      // [nph][C][C]
    const double* A;
    int nph;
    int lc = 0;           // batch entries per RVE (0: one RVE shared by all)
    long long mstride = 0;
};
// W consecutive voxels per item: with two in FP32 the global accesses are 8
// bytes a lane and a tile access a whole 16-byte pair of complex elements
template <typename T, int W_, int C = 6>
struct MidEM {
    static constexpr int NSUM = 1, W = W_;
    static constexpr bool kOne = false;
    typedef T Tr;  // type of the transforms
    typedef MidEMArgs<T> Args;
    Args a;
    long long V;
    struct Coef { T al, as, pl, ps; };
    static constexpr size_t smem_bytes(int nph) { return nph * sizeof(Coef); }
    const Coef* sm = nullptr;
    const uint8_t* phb = nullptr;
    T* xb = nullptr;
    const float* rb = nullptr;
    __device__ __forceinline__ void bind(int b) {
        V = a.V;
        phb = a.phase + (a.lc ? (long long)(b / a.lc) * V : 0);
        xb = a.x + (long long)b * C * V;
        rb = a.r ? a.r + (long long)b * C * V : nullptr;
    }
    __device__ __forceinline__ void load_smem(char* s, int b) {
        Coef* c = (Coef*)s;
        const long long o = a.lc ? (long long)(b / a.lc) * a.mstride : 0;
        for (int i = threadIdx.x; i < a.nph; i += blockDim.x) {
            const double *A = a.A + o + i * C * C, *P = a.P + o + i * C * C;
            if constexpr (C == 6) c[i] = Coef{(T)A[1], (T)A[21], (T)P[1], (T)P[21]};
            else c[i] = Coef{(T)0, (T)A[0], (T)0, (T)P[0]};
        }
        sm = c;
    }
    struct In {
        int p[W];
        T x[C][W];
        float r[C][W];
    };
    template <bool MIX> __device__ __forceinline__ void load(long long v, In& q) const {
        if constexpr (W == 2) {
            const uchar2 u = *reinterpret_cast<const uchar2*>(phb + v);
            q.p[0] = u.x;
            q.p[1] = u.y;
        } else {
            q.p[0] = phb[v];
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if constexpr (W == 2) {
                const float2 u = *reinterpret_cast<const float2*>(xb + c * V + v);
                q.x[c][0] = u.x;
                q.x[c][1] = u.y;
            } else {
                q.x[c][0] = xb[c * V + v];
            }
            if constexpr (MIX) {
                if constexpr (W == 2) {
                    const float2 u = rb ? *reinterpret_cast<const float2*>(rb + c * V + v) : make_float2(0.f, 0.f);
                    q.r[c][0] = u.x;
                    q.r[c][1] = u.y;
                } else {
                    q.r[c][0] = rb ? rb[c * V + v] : 0.f;
                }
            }
        }
    }
    // f: in the transform's values x_c of W voxels, out their polarization
    template <bool MIX> __device__ __forceinline__ void apply(const In& q, long long v, T (&f)[C][W], double* acc) const {
        T xn[C][W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const Coef k = sm[q.p[w]];
            if constexpr (MIX) {
                T d[C];
#pragma unroll
                for (int c = 0; c < C; ++c) d[c] = (f[c][w] + (T)q.r[c][w]) - q.x[c][w];
                double rs = 0;
#pragma unroll
                for (int c = 0; c < C; ++c) rs += (c < 3 ? 1.0 : 2.0) * (double)d[c] * (double)d[c];
                acc[0] += rs;
                const T tr = C == 6 ? k.al * (d[0] + d[1] + d[2]) : (T)0;
#pragma unroll
                for (int c = 0; c < C; ++c) xn[c][w] = q.x[c][w] + (C == 6 && c < 3 ? k.as * d[c] + tr : k.as * d[c]);
            } else {
#pragma unroll
                for (int c = 0; c < C; ++c) xn[c][w] = q.x[c][w];
            }
            const T tp = C == 6 ? k.pl * (xn[0][w] + xn[1][w] + xn[2][w]) : (T)0;
#pragma unroll
            for (int c = 0; c < C; ++c) f[c][w] = C == 6 && c < 3 ? k.ps * xn[c][w] + tp : k.ps * xn[c][w];
        }
        if constexpr (MIX) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if constexpr (W == 2) *reinterpret_cast<float2*>(xb + c * V + v) = make_float2(xn[c][0], xn[c][1]);
                else xb[c * V + v] = xn[c][0];
            }
        }
    }
};

// J2 / damage update of the basic scheme and the stress it transforms next (as
// EpiConstitutive followed by ProStress, inelastic.cuh).  The stress field
// itself is not stored: nothing between two sweeps reads it, and the end of an
// increment evaluates it once (k_constitutive) -- 48 of 249 bytes a voxel.
// The terms of C e are those of an isotropic C that are not 0, added in the order
// j2_update and damage_update add them, so that a voxel's update rounds as it does
// there.  (C e = la tr(e) I + 2 mu e left J2 strains 15% and plastic strains 20% further
// from the 64-bit results after one load step at 32^3, the mean of ten RVEs, for the
// same time.)  The von Mises value takes one square root and a product by 1/3: as close as
// vonmises(), which took 1 to 3% more of an FP32 solve.  Sums as
// EpiConstitutive: stress (6), strain (6), |d eps|^2.
struct MidJ2Args {
    const uint8_t* phase;
    double* eps;
    const double* eps_old;
    const double* sig_old;
    const double* ep;  // equivalent plastic strain (J2)
    double* dmg;       // damage (ed)
    long long V;
    const PhaseMech* ph;
    int nph;
    int increment;     // 1: the transform takes the stress increment of the load step
    int* nr_fail;
};
template <typename T, bool J2>
struct MidJ2 {
    static constexpr int NSUM = 13, W = 1;
    static constexpr bool kOne = true;  // one voxel at a time: 19 inputs
    typedef T Tr;
    typedef MidJ2Args Args;
    Args a;
    long long V;
    struct Coef { double cd, la, mu2, mu, Sy, H, n, P, Y0; };  // cd, la, mu2: C11, C12, C44
    static constexpr size_t smem_bytes(int nph) { return nph * sizeof(Coef); }
    const Coef* sm = nullptr;
    double *eb = nullptr, *db = nullptr;
    const double *eob = nullptr, *sob = nullptr, *epb = nullptr;
    __device__ __forceinline__ void bind(int b) {
        V = a.V;
        const long long o6 = (long long)b * 6 * V, o1 = (long long)b * V;
        eb = a.eps + o6;
        if constexpr (J2) {
            eob = a.eps_old + o6;
            sob = a.sig_old + o6;
            epb = a.ep + o1;
        } else {
            db = a.dmg + o1;
        }
    }
    __device__ __forceinline__ void load_smem(char* s, int) {
        Coef* c = (Coef*)s;
        for (int i = threadIdx.x; i < a.nph; i += blockDim.x) {
            const PhaseMech& p = a.ph[i];
            c[i] = Coef{p.C[0], p.C[1], p.C[21], p.mu, p.Sy, p.H, p.n, p.P, p.Y0};
        }
        sm = c;
    }
    // (C a)_i
    __device__ __forceinline__ static double mul(const Coef& k, const double (&a)[6], int i) {
        if (i >= 3) return k.mu2 * a[i];
        double s = (i == 0 ? k.cd : k.la) * a[0];
        s += (i == 1 ? k.cd : k.la) * a[1];
        s += (i == 2 ? k.cd : k.la) * a[2];
        return s;
    }
    struct In {
        int k;
        double e[6], eo[J2 ? 6 : 1], so[J2 ? 6 : 1], ep;
    };
    template <bool MIX> __device__ __forceinline__ void load(long long v, In& q) const {
        q.k = a.phase[v];
#pragma unroll
        for (int c = 0; c < 6; ++c) q.e[c] = eb[c * V + v];
        if constexpr (J2) {
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                q.eo[c] = eob[c * V + v];
                q.so[c] = sob[c * V + v];
            }
            q.ep = epb[v];
        } else {
            q.ep = db[v];
        }
    }
    template <bool MIX> __device__ __forceinline__ void apply(const In& q, long long v, T (&f)[6][1], double* acc) const {
        const Coef& k = sm[q.k];
        double e[6], sg[6], dd = 0;
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const double inc = MIX ? (double)f[c][0] : 0.0;
            e[c] = q.e[c] + inc;
            dd += (c >= 3 ? 2.0 : 1.0) * inc * inc;
        }
        if constexpr (J2) {
            double de[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) de[c] = e[c] - q.eo[c];
#pragma unroll
            for (int c = 0; c < 6; ++c) sg[c] = q.so[c] + mul(k, de, c);
            double sd[6];
            const double sm3 = (sg[0] + sg[1] + sg[2]) * (1.0 / 3.0);
#pragma unroll
            for (int c = 0; c < 6; ++c) sd[c] = c < 3 ? sg[c] - sm3 : sg[c];
            const double seff = sqrt(1.5 * (sd[0] * sd[0] + sd[1] * sd[1] + sd[2] * sd[2] +
                                            2 * (sd[3] * sd[3] + sd[4] * sd[4] + sd[5] * sd[5])));
            const double x = j2_multiplier(seff, q.ep, k.mu, k.Sy, k.H, k.n, a.nr_fail);
            if (x != 0.0) {  // sig -= (1.5 x / seff) C sd
                const double g = 1.5 * x / seff;
#pragma unroll
                for (int c = 0; c < 6; ++c) sg[c] -= g * mul(k, sd, c);
            }
        } else {
            double ce[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) ce[c] = mul(k, e, c);
            const double Y = sqrt(ce[0] * e[0] + ce[1] * e[1] + ce[2] * e[2] + 2 * ce[3] * e[3] + 2 * ce[4] * e[4] +
                                  2 * ce[5] * e[5]);
            double d = q.ep;
            if (Y > k.Y0) d = fmax(1 - exp(-k.P * (Y - k.Y0)), d);
#pragma unroll
            for (int c = 0; c < 6; ++c) sg[c] = (1 - d) * ce[c];
            if constexpr (MIX) db[v] = d;
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            if constexpr (MIX) {
                eb[c * V + v] = e[c];
                acc[c] += sg[c];
                acc[6 + c] += e[c];
            }
            f[c][0] = (T)(J2 && a.increment ? sg[c] - q.so[J2 ? c : 0] : sg[c]);
        }
        if constexpr (MIX) acc[12] += dd;
    }
};

}  // namespace m3d
