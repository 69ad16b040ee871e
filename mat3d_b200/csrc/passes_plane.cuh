// passes_plane.cuh -- two-pass sweeps of the six-component elastic operators:
// the kz-plane pass and the z-mid pass.
//
// The five-pass sweep moves each component's half spectrum through memory
// eight times and the state three times.  Here a sweep is two kernels:
//
//   k_plane  one kz plane (N x N modes of all six components): y FFT, x FFT,
//            Green operator, x inverse, y inverse, in shared memory
//   k_zmid   a group of z lines of all six components: z inverse (C2R), EM
//            update of the state and the residual partials, polarization of
//            the new state, z forward (R2C)         (+ fused finalize)
//
// so the spectrum crosses memory four times and the state is read and written
// once.  As in the slab sweep the forward half of k_zmid is speculative: when
// the finalize stops an entry, the spectrum it wrote is never read.
//
// Between the two kernels the half spectrum is stored plane by plane,
//     s[((b*6 + c)*Hz + kz)*N*N + x*N + y],   kz < Hz = N/2 + 1,
// (no larger than the row layout of passes.cuh, in the same buffer): a plane
// is one contiguous block, and k_zmid reads and writes runs of consecutive y.
// Lines, twiddles and Hermitian conventions are those of the five-pass
// kernels (the imaginary parts of kz = 0 and kz = N/2 are dropped in the C2R);
// fields agree with theirs to rounding.
//
// A plane of all six components has 6 N^2 complex values: 49 KB at FP32 32^2,
// 110 KB at 48^2, 197 KB at 64^2, 442 KB at 96^2.  Where two CTAs of all six
// no longer fit an SM, a cluster of CTAs shares them (CPC components per CTA)
// and the Green operator, which needs the six components of a mode together,
// reads and writes the other CTAs' planes through distributed shared memory.
//
// Measured per sweep (CUDA events; five passes -> k_plane + k_zmid):
//   FP32 96^3, 24 entries   1362 -> 440 + 388 us (the two kernels' bytes take
//                           162 + 390 us at the copy bandwidth)
//   FP32 64^3, 48 entries    912 -> 204 + 242 us
//   FP32 48^3, 96 entries    705 -> 183 + 215 us
//   FP32 32^3, 144 entries   386 ->  79 + 110 us
//   FP64 64^3, 1 entry        89 ->  27 +  25 us (with 10 us of event gaps)
// k_zmid runs at the memory bandwidth from 48^3 on; k_plane is bound by the
// shared-memory pipe (67% busy at 96^3: 16 accesses of a point in shared
// memory, the rows' global accesses in 32-byte pieces) and by issue (45%).
// FP64 96^3 (147 KB a component) has the four passes of passes_zmid.cuh.
#pragma once
#include <cooperative_groups.h>

#include "line_at.cuh"
#include "mid_ops.cuh"

namespace m3d {

template <typename T, int N> struct PlaneGeom {
    static constexpr bool ok = false;
};
#define M3D_PLANE(TY, NN, CPC_, NT_, MINB_)                                                     \
    template <> struct PlaneGeom<TY, NN> {                                                      \
        static constexpr bool ok = true;                                                        \
        static constexpr int CPC = CPC_, CS = 6 / CPC_, NT = NT_, MINB = MINB_, NW = NT_ / 32;  \
        static constexpr size_t smem() { return (size_t)(CPC * NN * NN + NN) * 2 * sizeof(TY); } \
    };
// components per CTA, threads, CTAs per SM.  Others, us per k_plane launch (these ->
// other): FP32 32^3 x 144 entries 77 -> 85 (3, 128, 8), 80 (6, 192, 4); 48^3 x 96 169 ->
// 166 (3, 192, 4), 169 (6, 256, 2); 64^3 x 48 193 -> 189 (6, 512, 1), 220 (2, 192, 3); 96^3
// x 24 411 -> 480 (2, 384, 1), 454 (1, 256, 3).  FP64, one entry and 96, 48 or 24: 32^3 18
// and 91 -> 16 and 96 (3, 128, 4), 19 and 94 (6, 384, 2); 48^3 25 and 186 -> 35 and 207
// (6, 512, 1), 21 and 184 (2, 192, 3); 64^3 28 and 221 -> 27 and 277 (2, 256, 1), 29 and
// 229 (1, 192, 3).
M3D_PLANE(float, 32, 6, 256, 4)
M3D_PLANE(float, 48, 6, 384, 2)
M3D_PLANE(float, 64, 3, 256, 2)
M3D_PLANE(float, 96, 1, 192, 3)
M3D_PLANE(double, 32, 6, 256, 2)
M3D_PLANE(double, 48, 3, 256, 2)
M3D_PLANE(double, 64, 1, 128, 3)
#undef M3D_PLANE

// Bank layout of a plane: element (row x, column y) sits at x*N + (y ^ f(x)),
// f of the row's two low bits.  The line FFTs exchange element (k1, t) of a
// line through its own storage, at index k1*T + (t ^ k1/Q): together every
// access of a warp -- rows and columns, natural, spectral and both exchange
// patterns -- touches each bank once.  Spectra are left in the order the lanes
// hold them (index t + T*r holds mode spec_mode(t, r)), which no one but the
// Green operator needs to know.
template <typename T> __device__ __forceinline__ int plane_swz(int row) {
    return sizeof(T) == 4 ? (((row & 1) << 3) | ((row & 2) << 1)) : ((row & 1) << 2);
}

// -G(xi) of one mode as SpecGreen, with one reciprocal for both schemes
template <typename T>
__device__ __forceinline__ void plane_green(int kind, T p1, T p2, T x0, T x1, T x2, T inv, const T (&t)[6], T (&o)[6]) {
    const T q0 = t[0] * x0 + t[5] * x1 + t[4] * x2;
    const T q1 = t[5] * x0 + t[1] * x1 + t[3] * x2;
    const T q2 = t[4] * x0 + t[3] * x1 + t[2] * x2;
    const T s = (x0 * q0 + x1 * q1 + x2 * q2) * inv;
    if (kind == GREEN_STRAIN) {
        // out_ij = -[ p1 (xi_j q_i + xi_i q_j)/|xi|^2 - p2 s xi_i xi_j/|xi|^2 ] = xi_i h_j + xi_j h_i
        const T a = -p1 * inv, bb = (T)0.5 * p2 * s * inv;
        const T h0 = a * q0 + bb * x0, h1 = a * q1 + bb * x1, h2 = a * q2 + bb * x2;
        o[0] = (T)2 * x0 * h0;
        o[1] = (T)2 * x1 * h1;
        o[2] = (T)2 * x2 * h2;
        o[3] = x1 * h2 + x2 * h1;
        o[4] = x0 * h2 + x2 * h0;
        o[5] = x0 * h1 + x1 * h0;
    } else {
        // P = I - n n^T: out_ij = -[ c3 P_ij (P:tau) + c4x2 (P tau P)_ij ]
        //   = -c4x2 tau_ij - c3 ptr delta_ij + xi_i h_j + xi_j h_i
        const T ptr = p1 * ((t[0] + t[1] + t[2]) - s);
        const T a = p2 * inv, bb = (T)0.5 * inv * (ptr - p2 * s);
        const T h0 = a * q0 + bb * x0, h1 = a * q1 + bb * x1, h2 = a * q2 + bb * x2;
        o[0] = (T)2 * x0 * h0 - (p2 * t[0] + ptr);
        o[1] = (T)2 * x1 * h1 - (p2 * t[1] + ptr);
        o[2] = (T)2 * x2 * h2 - (p2 * t[2] + ptr);
        o[3] = x1 * h2 + x2 * h1 - p2 * t[3];
        o[4] = x0 * h2 + x2 * h0 - p2 * t[4];
        o[5] = x0 * h1 + x1 * h0 - p2 * t[5];
    }
}

template <typename T, int N>
__global__ void __launch_bounds__(PlaneGeom<T, N>::NT, PlaneGeom<T, N>::MINB)
    k_plane(GridDims g, const typename Cx<T>::t* __restrict__ twx, typename Cx<T>::t* __restrict__ spec,
            SpecGreen<T, 6> op, const Ctl* __restrict__ ctl) {
    typedef typename Cx<T>::t C2;
    typedef PlaneGeom<T, N> P;
    constexpr int E = LineSplit<T, N>::E, TL = LineSplit<T, N>::Tl, LPW = 32 / TL, Q = E / TL;
    constexpr int CPC = P::CPC, CS = P::CS, NW = P::NW, NN = N * N, Hz = N / 2 + 1;
    const int b = entry_of(g, blockIdx.y);
    if (b < 0 || ctl[b].done) return;  // the same for every CTA of a cluster
    extern __shared__ __align__(16) char smem_raw[];
    C2* S = (C2*)smem_raw;  // [CPC][N][N]
    C2* tw = S + CPC * NN;
    const int kz = blockIdx.x / CS, rank = blockIdx.x - kz * CS;
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = twx[i];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // component c of this CTA: plane rank*CPC + c of the entry
    C2* gp = spec + (((long long)b * 6 + rank * CPC) * Hz + kz) * NN;
    __syncthreads();
    {   // y forward: rows, straight from global memory
        const int t = lane % TL, lw = lane / TL, sz = plane_swz<T>(lw);
#pragma unroll 1
        for (int l0 = warp * LPW; l0 < CPC * N; l0 += NW * LPW) {
            const int c = l0 / N, row = l0 - c * N + lw;
            const C2* src = gp + (long long)c * Hz * NN + row * N;
            C2* base = S + c * NN + row * N;
            C2 v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = src[t + TL * j];
            auto at = [&](int k1, int u) { return base + ((k1 * TL + u) ^ sz); };
            line_fwd_at<C2, E, TL>(v, t, tw, at);
#pragma unroll
            for (int r = 0; r < E; ++r) base[(t + TL * r) ^ sz] = v[r];
        }
    }
    __syncthreads();
    const int col = lane % LPW, tc = lane / LPW;
    {   // x forward: columns
#pragma unroll 1
        for (int gi = warp; gi < CPC * (N / LPW); gi += NW) {
            const int c = gi / (N / LPW), y = (gi - c * (N / LPW)) * LPW + col;
            C2* base = S + c * NN;
            auto at = [&](int k1, int u) { return base + (k1 * TL + u) * N + (y ^ plane_swz<T>(u)); };
            C2 v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = *at(j, tc);
            line_fwd_at<C2, E, TL>(v, tc, tw, at);
#pragma unroll
            for (int r = 0; r < E; ++r) *at(r, tc) = v[r];
        }
    }
    if constexpr (CS > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
    {   // Green operator, one mode per thread and step; the modes are dealt to the CTAs of the cluster
        op.prepare(ctl, b);
        C2* pl[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            if constexpr (CS > 1)
                pl[c] = cooperative_groups::this_cluster().map_shared_rank(S, c / CPC) + (c % CPC) * NN;
            else
                pl[c] = S + c * NN;
        }
        const T f0 = (T)sfreq(kz, (N - 1) / 2, N);
#pragma unroll 1
        for (int p = rank * P::NT + threadIdx.x; p < NN; p += CS * P::NT) {
            const int px = p / N, py = p - px * N;
            const int slot = px * N + (py ^ plane_swz<T>(px));
            C2 m[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) m[c] = pl[c][slot];
            // position t + TL r holds mode spec_mode(t, r)
            const int mx = spec_mode<E, TL>(px % TL, px / TL), my = spec_mode<E, TL>(py % TL, py / TL);
            if (kz == 0 && mx == 0 && my == 0) {
#pragma unroll
                for (int c = 0; c < 6; ++c) m[c] = mk<C2>(op.zero_k0 ? (T)0 : (T)ctl[b].kzero[c], (T)0);
            } else {
                const T f1 = (T)sfreq(my, (N - 1) / 2, N), f2 = (T)sfreq(mx, (N - 1) / 2, N);
                const T inv = (T)1 / (f0 * f0 + f1 * f1 + f2 * f2);
                T re[6], im[6], ore[6], oim[6];
#pragma unroll
                for (int c = 0; c < 6; ++c) { re[c] = m[c].x; im[c] = m[c].y; }
                plane_green<T>(op.kind, op.p1, op.p2, f0, f1, f2, inv, re, ore);
                plane_green<T>(op.kind, op.p1, op.p2, f0, f1, f2, inv, im, oim);
#pragma unroll
                for (int c = 0; c < 6; ++c) m[c] = mk<C2>(ore[c], oim[c]);
            }
#pragma unroll
            for (int c = 0; c < 6; ++c) pl[c][slot] = m[c];
        }
    }
    if constexpr (CS > 1) cooperative_groups::this_cluster().sync();  // also: no CTA leaves while others use its planes
    else __syncthreads();
    {   // x inverse
#pragma unroll 1
        for (int gi = warp; gi < CPC * (N / LPW); gi += NW) {
            const int c = gi / (N / LPW), y = (gi - c * (N / LPW)) * LPW + col;
            C2* base = S + c * NN;
            auto at = [&](int k1, int u) { return base + (k1 * TL + u) * N + (y ^ plane_swz<T>(u)); };
            C2 v[E];
#pragma unroll
            for (int r = 0; r < E; ++r) v[r] = *at(r, tc);
            line_inv_at<C2, E, TL>(v, tc, tw, at);
#pragma unroll
            for (int j = 0; j < E; ++j) *at(j, tc) = v[j];
        }
    }
    __syncthreads();
    {   // y inverse, straight to global memory
        const int t = lane % TL, lw = lane / TL, sz = plane_swz<T>(lw);
#pragma unroll 1
        for (int l0 = warp * LPW; l0 < CPC * N; l0 += NW * LPW) {
            const int c = l0 / N, row = l0 - c * N + lw;
            C2* dst = gp + (long long)c * Hz * NN + row * N;
            C2* base = S + c * NN + row * N;
            C2 v[E];
#pragma unroll
            for (int r = 0; r < E; ++r) v[r] = base[(t + TL * r) ^ sz];
            auto at = [&](int k1, int u) { return base + ((k1 * TL + u) ^ sz); };
            line_inv_at<C2, E, TL>(v, t, tw, at);
#pragma unroll
            for (int j = 0; j < E; ++j) dst[t + TL * j] = v[j];
        }
    }
    (void)Q;
}

// ---------------------------------------------------------------------------
// z-mid pass
// ---------------------------------------------------------------------------
// G lines (consecutive y) of six components: 3 G complex lines, each the pair
// (2p, 2p+1) of a voxel line, row p*G + gi of the tile; a warp owns eight lines
// of one pair, so it loads, transforms, splits and stores its rows without a
// block barrier and only the pointwise step needs the whole tile.  G = 8, and
// 16 at N = 32, where eight lines are too little work for a CTA.
//
// Bank layout.  Every length is split N = E x 4 here (lane t = lane mod 4).
// Rows are N + 4 elements, a quarter of a bank cycle apart, and spectra lie in
// the order the lanes hold them: mode k = t Q + q + E k2 (q < Q = E/4, k2 < 4)
// at 16 q + 4 k2 + t.  With the exchange of line_fwd_at, natural, spectral and
// exchange accesses all touch each bank once, the loads and stores of the half
// spectra too (their lanes are dealt 4 rows x 4 modes; FP64: 2 x 4).  Before
// the inverse transform the free k2 = 2, 3 places of the pair's first spectrum
// hold the second (mode k at + 8), the two Nyquist values the places N, N + 1.
// With natural order and rows of N + 36 a third of the shared-memory wavefronts
// were conflicts and the data pipe was 79% busy at FP32 96^3.
template <typename T, int N> struct ZMidGeom {
    static constexpr int TL = 4, E = N / 4, Q = E / 4, LPW = 8;
    static constexpr int G = N == 32 ? 16 : 8, WPP = G / 8, LINES = 3 * G, NT = 96 * WPP, ROW = N + 4, Hz = N / 2 + 1;
    // voxels per item: a thread's 2.67 voxels at N = 32 divide better singly
    static constexpr int W = sizeof(T) == 4 && N > 32 ? 2 : 1;
    static constexpr int ITEMS = G * N / W, PER = (ITEMS + NT - 1) / NT;
    static constexpr int PF = PER < (sizeof(T) == 4 ? 2 : 3) ? PER : (sizeof(T) == 4 ? 2 : 3);  // loaded before the transform
    // CTAs per SM: 15 warps of 128 registers in FP32 (18 of 112 at N = 32), 9 of 168 in FP64
    static constexpr int MINB = WPP == 2 ? (sizeof(T) == 4 ? 3 : 1) : (sizeof(T) == 4 ? 5 : 3);
    static_assert(N % 16 == 0, "N = 16 Q");
    static constexpr size_t smem() {
        return (size_t)N * 2 * sizeof(T) + (size_t)LINES * ROW * 2 * sizeof(T) + 64 * sizeof(double) + kMaxPhases * 4 * sizeof(T);
    }
};

template <typename T, int N, class Op, bool MIX, class Fin>
__global__ void __launch_bounds__(ZMidGeom<T, N>::NT, ZMidGeom<T, N>::MINB)
    k_zmid(GridDims g, const typename Cx<T>::t* __restrict__ twz, typename Cx<T>::t* __restrict__ spec,
           typename Op::Args args, Ctl* ctl, double* partials, Fin fin) {
    typedef typename Cx<T>::t C2;
    typedef ZMidGeom<T, N> Z;
    constexpr int E = Z::E, TL = Z::TL, Q = Z::Q, G = Z::G, ROW = Z::ROW, Hz = Z::Hz, NN = N * N, W = Z::W;
    const int b = entry_of(g, blockIdx.y);
    if (b < 0 || ctl[b].done) return;
    Op op;
    op.a = args;
    op.bind(b);
    extern __shared__ __align__(16) char smem_raw[];
    C2* tw = (C2*)smem_raw;
    C2* tile = tw + N;
    double* red = (double*)(tile + Z::LINES * ROW);
    const int x = blockIdx.x / (N / G), y0 = (blockIdx.x - x * (N / G)) * G;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = lane % TL;
    C2* row = tile + (warp * 8 + lane / TL) * ROW;  // this lane's line
    auto at = [&](int k1, int u) { return row + k1 * TL + u; };
    // half spectra of the warp's pair: row li, modes kk Q + q + E k2
    const int li = sizeof(T) == 4 ? ((lane & 3) | ((lane >> 4) << 2)) : ((lane & 1) | ((lane >> 3) << 1));
    const int kk = sizeof(T) == 4 ? ((lane >> 2) & 3) : ((lane >> 1) & 3);
    C2* sb = spec + ((long long)b * 6 + 2 * (warp / Z::WPP)) * Hz * NN + x * N + y0 + (warp % Z::WPP) * 8 + li;
    C2* rl = tile + (warp * 8 + li) * ROW;
    if constexpr (MIX) {
        const C2* sk = sb + (long long)kk * Q * NN;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k2 = 0; k2 < 2; ++k2)
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    cp_async_c(rl + 16 * q + 4 * k2 + 8 * h + kk, sk + (long long)(h * Hz + q + E * k2) * NN);
        if (kk < 2) cp_async_c(rl + N + kk, sb + (long long)(kk * Hz + 2 * E) * NN);
    }
    // the state's loads do not depend on the transform: the first of them before it
    const long long v0 = ((long long)x * N + y0) * N;  // the tile's voxels are contiguous
    typename Op::In in[Z::PF];
#pragma unroll
    for (int k = 0; k < Z::PF; ++k) {
        const int i = threadIdx.x + k * Z::NT;
        if (i < Z::ITEMS) op.template load<MIX>(v0 + W * i, in[k]);
    }
    for (int i = threadIdx.x; i < N; i += Z::NT) tw[i] = twz[i];
    op.load_smem((char*)(red + 64), b);
    if constexpr (MIX) cp_async_wait_all();
    __syncthreads();
    if constexpr (MIX) {
        // z inverse: the pair's spectrum a + i b assembled from the two half
        // spectra as the lanes load it (Hermitian extension: mode N - k is
        // conj a + i conj b of mode k; k = 0 and N/2 keep their real parts)
        C2 v[E];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) {
                // place of mode k (k2 < 2) or N - k
                int pos;
                if (k2 < 2) pos = 16 * q + 4 * k2 + t;
                else if (q > 0) pos = 16 * (Q - q) + 4 * (3 - k2) + 3 - t;
                else pos = t > 0 ? 4 * (3 - k2) + 4 - t : (k2 == 2 ? N : 4);
                const bool nyq = q == 0 && k2 == 2 && t == 0;
                const C2 a = row[pos], s = row[nyq ? N + 1 : pos + 8];
                if (k2 < 2) v[q * 4 + k2] = mk<C2>(a.x - s.y, a.y + s.x);
                else v[q * 4 + k2] = mk<C2>(a.x + s.y, s.x - a.y);
                if (q == 0 && (k2 == 0 || k2 == 2) && t == 0) v[q * 4 + k2] = mk<C2>(a.x, s.x);
            }
        }
        line_inv_at<C2, E, TL>(v, t, tw, at);
#pragma unroll
        for (int j = 0; j < E; ++j) row[t + TL * j] = v[j];
        __syncthreads();
    }
    const T invV = (T)(1.0 / (double)g.V);
    double acc[Op::NSUM] = {};
    auto point = [&](int i, const typename Op::In& q) {
        const int gi = i / (N / W), z = W * (i - gi * (N / W));
        C2* tp = tile + gi * ROW + z;
        T f[6][W];
        if constexpr (MIX) {
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                C2 u[W];
                tile_get(tp + p * G * ROW, u);
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    f[2 * p][w] = u[w].x * invV;
                    f[2 * p + 1][w] = u[w].y * invV;
                }
            }
        }
        op.template apply<MIX>(q, v0 + W * i, f, acc);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            C2 u[W];
#pragma unroll
            for (int w = 0; w < W; ++w) u[w] = mk<C2>(f[2 * p][w], f[2 * p + 1][w]);
            tile_put(tp + p * G * ROW, u);
        }
    };
    {
        typename Op::In rest[Z::PER - Z::PF > 0 ? Z::PER - Z::PF : 1];
#pragma unroll
        for (int k = Z::PF; k < Z::PER; ++k) {
            const int i = threadIdx.x + k * Z::NT;
            if (i < Z::ITEMS) op.template load<MIX>(v0 + W * i, rest[k - Z::PF]);
        }
#pragma unroll
        for (int k = 0; k < Z::PER; ++k) {
            const int i = threadIdx.x + k * Z::NT;
            if (i < Z::ITEMS) point(i, k < Z::PF ? in[k < Z::PF ? k : 0] : rest[k < Z::PF ? 0 : k - Z::PF]);
        }
    }
    __syncthreads();
    {   // z forward, split into the pair's half spectra as they are stored
        C2 v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = row[t + TL * j];
        line_fwd_at<C2, E, TL>(v, t, tw, at);
#pragma unroll
        for (int r = 0; r < E; ++r) row[t + TL * r] = v[r];
        __syncwarp();
        C2* sk = sb + (long long)kk * Q * NN;
        auto split = [&](C2* d, C2 Zk, C2 Zm) {
            d[0] = mk<C2>((T)0.5 * (Zk.x + Zm.x), (T)0.5 * (Zk.y - Zm.y));
            d[(long long)Hz * NN] = mk<C2>((T)0.5 * (Zk.y + Zm.y), (T)-0.5 * (Zk.x - Zm.x));
        };
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2)
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                int m;  // place of mode N - k
                if (q > 0) m = 16 * (Q - q) + 4 * (3 - k2) + 3 - kk;
                else m = kk > 0 ? 4 * (3 - k2) + 4 - kk : (k2 == 0 ? 0 : 12);
                split(sk + (long long)(q + E * k2) * NN, rl[16 * q + 4 * k2 + kk], rl[m]);
            }
        if (kk == 0) split(sb + (long long)(2 * E) * NN, rl[8], rl[8]);
    }
    if constexpr (MIX) {
        block_reduce_store<Op::NSUM>(acc, red, partials, b, gridDim.x, blockIdx.x);
        fused_finalize(fin, ctl, partials, Op::NSUM, b);
    }
}

}  // namespace m3d
