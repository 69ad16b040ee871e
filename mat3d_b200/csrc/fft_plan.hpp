// fft_plan.hpp -- host-side set-up of the generic line FFTs: the radix
// schedule of a length and its twiddle table (shared by the 3-D and 2-D solvers).
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft_smem.cuh"

namespace m3d {

// The radices of the factors 2, 3 and 5 with a register DFT; the primes above
// come one per stage.
constexpr int kRadices[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
// The fewest of kRadices (largest first) whose product is m, among those the
// smallest sum.
inline void fewest_radices(int m, std::vector<int>& cur, std::vector<int>& best, bool& have) {
    auto sum = [](const std::vector<int>& v) {
        int t = 0;
        for (int r : v) t += r;
        return t;
    };
    if (m == 1) {
        if (!have || cur.size() < best.size() || (cur.size() == best.size() && sum(cur) < sum(best))) best = cur;
        have = true;
        return;
    }
    if (have && cur.size() + 1 > best.size()) return;
    for (int r : kRadices)
        if (m % r == 0 && (cur.empty() || r <= cur.back())) {
            cur.push_back(r);
            fewest_radices(m / r, cur, best, have);
            cur.pop_back();
        }
}

// radix schedule of a length; false if a prime factor is above 31.  Any order
// and grouping of the factors is a valid Stockham schedule; `order` picks one
// for the autotuner: 0 as few stages as possible, the primes above 5 first
// (the first stage needs no twiddle multiplications, so the costliest
// butterfly goes there), then by radix; 1 one factor per stage, odd factors
// smallest first, then 8s, 4, 2; 2 the power-of-two stages first; 3 odd factors
// largest first, the power of two as radix-4 stages (and one 2).
// complex_lines (order 0; the reconstruction, whose fields' phases matter): odd radices
// first, so that the middle mode of an even line of real values comes out with an
// imaginary part of exactly 0 (its phase, 0 or pi, would else take the sign of a
// rounding error); and stages 6 and 3 as 9 and 2, 6 and 6 as 9 and 4, because the paired
// 9-point DFT of these kernels (fft_smem.cuh) rounds less: FP64 transforms of 18, 36,
// 126, 216 and 252 points 7, 2, 1, 6 and 3% nearer their exact values, for 5 to 8% of the
// time at 36, 126 and 162.
constexpr int kPlanOrders = 4;
inline bool make_plan(int n, LinePlan& p, int order = 0, bool complex_lines = false) {
    std::vector<int> f, odd;
    int m = n;
    int p2 = 0;
    while (m % 2 == 0) { ++p2; m /= 2; }
    for (int q = 3; q <= m; q += 2)
        while (m % q == 0) { odd.push_back(q); m /= q; }  // ascending
    if (order == 0) {
        int smooth = 1 << p2;
        for (size_t i = odd.size(); i-- > 0;)
            if (odd[i] > 5) f.push_back(odd[i]);
            else smooth *= odd[i];
        std::vector<int> cur, best;
        bool have = false;
        fewest_radices(smooth, cur, best, have);
        for (bool more = complex_lines; more;) {
            auto six = std::find(best.begin(), best.end(), 6);
            auto mate = six == best.end() ? six : std::find_if(six + 1, best.end(), [](int r) { return r == 6 || r == 3; });
            more = mate != best.end();
            if (!more) break;
            *mate = *mate == 6 ? 4 : 2;
            *six = 9;
            std::sort(best.rbegin(), best.rend());
        }
        if (complex_lines) std::stable_partition(best.begin(), best.end(), [](int r) { return r % 2 == 1; });
        f.insert(f.end(), best.begin(), best.end());
    } else {
        std::vector<int> pow2;
        if (order == 3) {
            for (; p2 >= 2; p2 -= 2) pow2.push_back(4);
        } else {
            for (; p2 >= 3; p2 -= 3) pow2.push_back(8);
            if (p2 == 2) pow2.push_back(4);
        }
        if (p2 == 1) pow2.push_back(2);
        if (order == 2) f = pow2;
        if (order == 1) f.insert(f.end(), odd.begin(), odd.end());
        else f.insert(f.end(), odd.rbegin(), odd.rend());
        if (order != 2) f.insert(f.end(), pow2.begin(), pow2.end());
    }
    if (f.empty()) f.push_back(1);
    if ((int)f.size() > kMaxStages) return false;
    for (int r : f)
        if (r > kMaxGenericRadix) return false;
    p.n = n;
    p.nstages = (n == 1) ? 0 : (int)f.size();
    for (int i = 0; i < kMaxStages; ++i) p.radix[i] = i < (int)f.size() ? f[i] : 1;
    finish_plan(p);
    return true;
}

// Threads of a CTA that transforms `lines` lines of plan p together: one per
// butterfly of its widest stage, 64 to `most`.
inline int plan_threads(const LinePlan& p, int lines, int most = 256) {
    int r = 1;
    for (int s = 0; s < p.nstages; ++s) r = std::max(r, p.radix[s]);
    const int b = lines * (p.n / r);
    return std::max(64, std::min(most, (b + 31) / 32 * 32));
}

// tw[m] = exp(-2 pi i m / n), evaluated in long double
template <typename T>
inline std::vector<typename Cx<T>::t> twiddles(int n) {
    std::vector<typename Cx<T>::t> t(n);
    const long double two_pi = 6.283185307179586476925286766559L;
    for (int m = 0; m < n; ++m) {
        const long double a = -two_pi * (long double)m / (long double)n;
        t[m].x = (T)cosl(a);
        t[m].y = (T)sinl(a);
    }
    return t;
}

}  // namespace m3d
