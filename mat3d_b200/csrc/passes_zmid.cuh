// passes_zmid.cuh -- the fused z pass of four-pass sweeps: z inverse, the
// pointwise middle of the sweep (mid_ops.cuh) and the next sweep's z forward in
// one kernel, on the row layout of the half spectrum (passes.cuh).
//
// A sweep is then x turnaround, y inverse, k_zmid_rows, y forward: the state is
// read once instead of twice, and the stress of the inelastic sweeps stays in
// registers.  The forward half is speculative, as in the two-pass sweeps.
// Measured, J2 (z forward + z inverse -> k_zmid_rows): FP64 256^3 2376 -> 1343 us,
// FP32 256^3 2671 -> 967, FP32 64^3 64 -> 44.  Bound by latency: 12 warps per SM
// of FP64 dependency chains (issue 24%, long scoreboard the largest stall); the
// bytes of a J2 voxel (201 and its share of the spectrum) take 765 us at FP64
// 256^3.  EM update, z forward + z inverse -> fused: FP32 thermal 256^3
// 173 + 394 -> 212 us (124 us of bytes), FP64 thermal 128^3 52 + 76 -> 68, FP64
// elastic 96^3 48 + 78 -> 54.
//
// CTAs of three warps walk tiles of G z lines of C components, C G/2 packed
// complex lines (lines y, y + 1 of one component), LPW per warp.  The next
// tile's spectra are copied into a second buffer while the current tile is
// worked on, where two buffers leave room for the CTAs per SM; and a solve has
// at most kZRowsGrid partial sums per entry, so that the last CTA's finalize
// stays short (an inelastic sweep has 13 sums: 32768 partials of each at 256^3,
// one per pair of lines, were half a millisecond of one CTA's reads).  The
// number of CTAs depends on the grid alone, so an entry's sums do not depend on
// the batch it runs in.  A warp loads, transforms,
// splits and stores its own lines; only the pointwise step, which needs all
// components of a voxel, takes block barriers.  Tile rows hold a spectrum in the
// order the lanes hold it: mode k = t Q + q + E k2 at T (q T + k2) + t; before
// the inverse transform the places k2 >= T/2 hold the second line's half
// spectrum (mode k at + T T/2), the places N, N + 1 the two Nyquist values.
#pragma once
#include "line_at.cuh"
#include "mid_ops.cuh"

namespace m3d {

template <typename T, int N> struct MidSplit { static constexpr int Tl = N >= 256 ? 16 : (N == 64 || N == 128 ? 8 : 4); };

template <typename T, int N, int C> struct ZRowsGeom {
    static constexpr int TL = MidSplit<T, N>::Tl, E = N / TL, Q = E / TL, LPW = 32 / TL;
    static constexpr int G = 6 * LPW / C, PL = 3 * LPW, NT = 96, PP = G / 2;  // packed lines per component
    static constexpr int Hz = N / 2 + 1, Hzp = HzOf<N>::Hzp;
    // rows a quarter (T = 4) or half (T = 8) bank cycle apart
    static constexpr int ROW = N + (TL == 8 ? 8 : 4);
    static_assert(N % G == 0 && E % TL == 0 && ROW >= N + 2, "whole groups of lines; room for the half spectra");
    static constexpr size_t tile_bytes = (size_t)PL * ROW * 2 * sizeof(T);
    static constexpr int NBUF = 2 * tile_bytes <= 52 * 1024 ? 2 : 1;
    static_assert(NBUF * tile_bytes >= 32 * 13 * sizeof(double), "the block reduction reuses the tile");
    template <class Op> static size_t smem(int nph) {
        return (size_t)N * 2 * sizeof(T) + NBUF * tile_bytes + Op::smem_bytes(nph);
    }
};
constexpr int kZRowsGrid = kSMs * 4;

// CTAs (of three warps) per SM: four, 168 registers.  The inelastic kernels spill
// 100-400 bytes under it; at 128 registers (five CTAs, one buffer) FP64 256^3
// took 1463 us against 1343, with one buffer and four CTAs 1355.
constexpr int kZRowsMinB = 4;

template <typename T, int N, int C, class Op, class Fin>
__global__ void __launch_bounds__(96, kZRowsMinB)
    k_zmid_rows(GridDims g, const typename Cx<T>::t* __restrict__ twz, typename Cx<T>::t* __restrict__ spec,
                typename Op::Args args, Ctl* ctl, double* partials, Fin fin) {
    typedef typename Cx<T>::t C2;
    typedef ZRowsGeom<T, N, C> Z;
    constexpr int E = Z::E, TL = Z::TL, Q = Z::Q, LPW = Z::LPW, G = Z::G, PP = Z::PP, ROW = Z::ROW, Hzp = Z::Hzp;
    constexpr int W = Op::W, H = N / 2;
    const int b = entry_of(g, blockIdx.y);
    if (b < 0 || ctl[b].done) return;
    Op op;
    op.a = args;
    op.bind(b);
    extern __shared__ __align__(16) char smem_raw[];
    C2* tw = (C2*)smem_raw;
    C2* buf = tw + N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = lane % TL;
    const int ntiles = (int)(g.NL / G);
    for (int i = threadIdx.x; i < N; i += Z::NT) tw[i] = twz[i];
    op.load_smem((char*)(buf + Z::NBUF * Z::PL * ROW), b);
    // packed line pl: component pl / PP, lines l0 + 2 (pl % PP) and + 1
    auto gline = [&](long long l0, int pl) {
        const int c = pl / PP, p = pl - c * PP;
        return spec + (((long long)b * C + c) * g.NL + l0 + 2 * p) * Hzp;
    };
    auto place = [&](int k) {  // of mode k in a spectrum
        if constexpr (Q == 1) return k;
        const int k2 = k / E, m = k - k2 * E, tt = m / Q, q = m - tt * Q;
        return TL * (q * TL + k2) + tt;
    };
    auto fetch = [&](C2* tile, long long l0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll 4
            for (int i = lane; i < LPW * H; i += 32) {
                const int ll = i / H, k = i - ll * H, pl = warp * LPW + ll;
                cp_async_c(tile + pl * ROW + place(k) + h * (TL * TL / 2), gline(l0, pl) + h * Hzp + k);
            }
        }
        if (lane < 2 * LPW) {
            const int pl = warp * LPW + (lane >> 1), h = lane & 1;
            cp_async_c(tile + pl * ROW + N + h, gline(l0, pl) + h * Hzp + H);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    double acc[Op::NSUM] = {};
    const T invV = (T)(1.0 / (double)g.V);
    if (Z::NBUF == 2) fetch(buf, (long long)blockIdx.x * G);
    __syncthreads();
    int cur = 0;
#pragma unroll 1
    for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
        const long long l0 = (long long)ti * G;
        C2* tile = buf + cur * (Z::PL * ROW);
        C2* row = tile + (warp * LPW + lane / TL) * ROW;  // this lane's packed line
        auto at = [&](int k1, int u) { return row + k1 * TL + u; };
        if (Z::NBUF == 1) fetch(tile, l0);
        // items: W voxels of each of the two lines of a pair, or (an operator of
        // many inputs) one voxel, the next one's inputs loaded meanwhile
        constexpr bool ONE = Op::kOne;
        constexpr int IPL = N / W, ITEMS = ONE ? G * N : PP * IPL, PER = (ITEMS + Z::NT - 1) / Z::NT;
        auto voxel = [&](int i) {
            if constexpr (ONE) return l0 * N + i;
            const int p = i / IPL, z = W * (i - p * IPL);
            return (l0 + 2 * p) * N + z;
        };
        typename Op::In pre[2];  // the first item's inputs, loaded before the transform
        op.template load<true>(voxel(threadIdx.x), pre[0]);  // (96 <= ITEMS)
        if constexpr (!ONE) op.template load<true>(voxel(threadIdx.x) + N, pre[1]);
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncwarp();
        if (Z::NBUF == 2) {  // its rows of the other buffer were last used before this warp's stores of the previous tile
            cur ^= 1;
            if (ti + (int)gridDim.x < ntiles) fetch(buf + cur * (Z::PL * ROW), l0 + (long long)gridDim.x * G);
        }
        {
            C2 v[E];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
#pragma unroll
                for (int k2 = 0; k2 < TL; ++k2) {
                    int pos;  // place of mode k (k2 < T/2) or N - k
                    if (k2 < TL / 2) pos = TL * (q * TL + k2) + t;
                    else if (q > 0) pos = TL * ((Q - q) * TL + TL - 1 - k2) + TL - 1 - t;
                    else pos = t > 0 ? TL * (TL - 1 - k2) + TL - t : (k2 == TL / 2 ? N : TL * (TL - k2));
                    const bool nyq = q == 0 && k2 == TL / 2 && t == 0;
                    const C2 a = row[pos], s = row[nyq ? N + 1 : pos + TL * TL / 2];
                    if (k2 < TL / 2) v[q * TL + k2] = mk<C2>(a.x - s.y, a.y + s.x);
                    else v[q * TL + k2] = mk<C2>(a.x + s.y, s.x - a.y);
                    if (q == 0 && (k2 == 0 || k2 == TL / 2) && t == 0) v[q * TL + k2] = mk<C2>(a.x, s.x);
                }
            }
            line_inv_at<C2, E, TL>(v, t, tw, at);
#pragma unroll
            for (int j = 0; j < E; ++j) row[t + TL * j] = v[j];
        }
        __syncthreads();
        if constexpr (ONE) {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = threadIdx.x + k * Z::NT;
                if (k + 1 < PER && i + Z::NT < ITEMS) op.template load<true>(voxel(i + Z::NT), pre[(k + 1) & 1]);
                if (i < ITEMS) {
                    const int gi = i / N, z = i - gi * N;
                    T* tp = (T*)(tile + (gi >> 1) * ROW + z) + (gi & 1);  // component c: + 2 c PP ROW
                    T f[C][1];
#pragma unroll
                    for (int c = 0; c < C; ++c) f[c][0] = tp[2 * c * PP * ROW] * invV;
                    op.template apply<true>(pre[k & 1], voxel(i), f, acc);
#pragma unroll
                    for (int c = 0; c < C; ++c) tp[2 * c * PP * ROW] = f[c][0];
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = threadIdx.x + k * Z::NT;
                if (i < ITEMS) {
                    const int p = i / IPL, z = W * (i - p * IPL);
                    C2* tp = tile + p * ROW + z;  // component c: + c PP ROW
                    const long long v0 = voxel(i);
                    if (k > 0) {
                        op.template load<true>(v0, pre[0]);
                        op.template load<true>(v0 + N, pre[1]);
                    }
                    T f[2][C][W];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        C2 u[W];
                        tile_get(tp + c * PP * ROW, u);
#pragma unroll
                        for (int w = 0; w < W; ++w) {
                            f[0][c][w] = u[w].x * invV;
                            f[1][c][w] = u[w].y * invV;
                        }
                    }
                    op.template apply<true>(pre[0], v0, f[0], acc);
                    op.template apply<true>(pre[1], v0 + N, f[1], acc);
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        C2 u[W];
#pragma unroll
                        for (int w = 0; w < W; ++w) u[w] = mk<C2>(f[0][c][w], f[1][c][w]);
                        tile_put(tp + c * PP * ROW, u);
                    }
                }
            }
        }
        __syncthreads();
        {
            C2 v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = row[t + TL * j];
            line_fwd_at<C2, E, TL>(v, t, tw, at);
#pragma unroll
            for (int r = 0; r < E; ++r) row[t + TL * r] = v[r];
        }
        __syncwarp();
        auto split = [&](C2* d, C2 Zk, C2 Zm) {
            d[0] = mk<C2>((T)0.5 * (Zk.x + Zm.x), (T)0.5 * (Zk.y - Zm.y));
            d[Hzp] = mk<C2>((T)0.5 * (Zk.y + Zm.y), (T)-0.5 * (Zk.x - Zm.x));
        };
#pragma unroll 4
        for (int i = lane; i < LPW * H; i += 32) {
            const int ll = i / H, k = i - ll * H, pl = warp * LPW + ll;
            const C2* r = tile + pl * ROW;
            split(gline(l0, pl) + k, r[place(k)], r[place(k == 0 ? 0 : N - k)]);
        }
        if (lane < LPW) {
            const int pl = warp * LPW + lane;
            const C2 z = tile[pl * ROW + place(H)];
            split(gline(l0, pl) + H, z, z);
        }
        if (Z::NBUF == 1) __syncwarp();  // the rows are refilled next
    }
    __syncthreads();
    double* red = (double*)buf;
    block_reduce_store<Op::NSUM>(acc, red, partials, b, gridDim.x, blockIdx.x);
    fused_finalize(fin, ctl, partials, Op::NSUM, b);
}

// ---------------------------------------------------------------------------
// The same for lengths without a compile-time transform (generic Stockham lines,
// fft_smem.cuh): CTAs walk tiles of G lines of all components, packed line
// p*C + c holding lines 2p, 2p + 1 of component c; one voxel per pointwise item.
// Measured, elastic 75^3 FP32, six entries: z forward 63 + z inverse 108 us ->
// 137.  Tiles as large as the separate passes' (48 KB): dealing a small grid to
// at least four tiles per SM made most sizes slower (homogenization of eight
// RVEs at 45^3 28.2 -> 36.9 ms).
// ---------------------------------------------------------------------------
template <typename T, int C, class Op, class Fin, int MaxR>
__global__ void __launch_bounds__(256)
    k_zmid_gen(GridDims g, const __grid_constant__ LinePlan pz, const typename Cx<T>::t* __restrict__ twz,
               typename Cx<T>::t* __restrict__ spec, typename Op::Args args, Ctl* ctl, int G, double* partials, Fin fin) {
    typedef typename Cx<T>::t C2;
    const int b = entry_of(g, blockIdx.y);
    if (b < 0 || ctl[b].done) return;
    Op op;
    op.a = args;
    op.bind(b);
    extern __shared__ __align__(16) char smem_raw[];
    const int Nz = g.Nz, Hz = g.Hz, Hzp = g.Hzp;
    const int nl = G / 2 * C;
    C2* tw = (C2*)smem_raw;
    C2* A = tw + Nz;
    C2* B = A + (size_t)nl * Nz;
    char* extra = align_up((char*)(B + (size_t)nl * Nz), 16);
    double* red = (double*)extra;
    for (int i = threadIdx.x; i < Nz; i += blockDim.x) tw[i] = twz[i];
    op.load_smem(extra + 32 * Op::NSUM * sizeof(double), b);
    const LineLayout L{nl, 1, 0, Nz, 1, false};
    const T invV = (T)(1.0 / (double)g.V);
    double acc[Op::NSUM] = {};
    const int ntiles = (int)((g.NL + G - 1) / G);
#pragma unroll 1
    for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
        const long long l0 = (long long)ti * G;
        for (int i = threadIdx.x; i < nl * Hz; i += blockDim.x) {
            const int pc = g.dHz.div(i), k = i - pc * Hz;
            const int p = pc / C, c = pc - p * C;
            const long long la = l0 + 2 * p;
            const C2* s = spec + (((long long)b * C + c) * g.NL + la) * Hzp + k;
            const C2 a = la < g.NL ? s[0] : mk<C2>(0, 0);
            const C2 q = la + 1 < g.NL ? s[Hzp] : mk<C2>(0, 0);
            C2* line = A + (size_t)pc * Nz;
            if (k == 0 || 2 * k == Nz) {
                line[k] = mk<C2>(a.x, q.x);
            } else {
                line[k] = mk<C2>(a.x - q.y, a.y + q.x);
                line[Nz - k] = mk<C2>(a.x + q.y, q.x - a.y);
            }
        }
        __syncthreads();
        C2* R = fft_lines<C2, MaxR>(A, B, tw, pz, L, +1);
        C2* S = R == A ? B : A;
        for (int i = threadIdx.x; i < G * Nz; i += blockDim.x) {
            const int gi = pz.dn.div(i), z = i - gi * Nz;
            const long long l = l0 + gi;
            T* t = (T*)R + 2 * ((size_t)(gi >> 1) * C * Nz + z) + (gi & 1);  // component c: + 2 c Nz
            T f[C][1];
            if (l < g.NL) {
                typename Op::In q;
                op.template load<true>(l * Nz + z, q);
#pragma unroll
                for (int c = 0; c < C; ++c) f[c][0] = t[2 * c * Nz] * invV;
                op.template apply<true>(q, l * Nz + z, f, acc);
            } else {
#pragma unroll
                for (int c = 0; c < C; ++c) f[c][0] = (T)0;
            }
#pragma unroll
            for (int c = 0; c < C; ++c) t[2 * c * Nz] = f[c][0];
        }
        __syncthreads();
        R = fft_lines<C2, MaxR>(R, S, tw, pz, L, -1);
        for (int i = threadIdx.x; i < nl * Hz; i += blockDim.x) {
            const int pc = g.dHz.div(i), k = i - pc * Hz;
            const int p = pc / C, c = pc - p * C;
            const long long la = l0 + 2 * p;
            C2* s = spec + (((long long)b * C + c) * g.NL + la) * Hzp + k;
            const C2 Z = R[(size_t)pc * Nz + k];
            const C2 Zm = R[(size_t)pc * Nz + (k == 0 ? 0 : Nz - k)];
            if (la < g.NL) s[0] = mk<C2>((T)0.5 * (Z.x + Zm.x), (T)0.5 * (Z.y - Zm.y));
            if (la + 1 < g.NL) s[Hzp] = mk<C2>((T)0.5 * (Z.y + Zm.y), (T)-0.5 * (Z.x - Zm.x));
        }
        __syncthreads();  // the next tile is loaded over this one
    }
    block_reduce_store<Op::NSUM>(acc, red, partials, b, gridDim.x, blockIdx.x);
    fused_finalize(fin, ctl, partials, Op::NSUM, b);
}
constexpr int kZGenGrid = kSMs * 8;  // CTAs per entry at most (partial sums, as kZRowsGrid)

}  // namespace m3d
