// longline.cuh -- x lines of a long prime length (47, 83, 97), shared among
// threads (host and device): the tasks of the LONG kernels.
//
// The folded sum of dft_odd_folded (codelets.cuh) over H = (N - 1)/2 conjugate
// pairs, KT of the H output pairs a task: the task runs once through the line in
// shared memory and adds each pair's sum and difference, times the factors of
// its own outputs, into 4 KT accumulators.  Lanes run along the lines, so a
// factor is one shared-memory broadcast.  Sums and factors are double in both
// precisions, as in pass_x_out_direct (volume.cuh).
#pragma once

#include "volume.cuh"

namespace fft3d {

template <class G_, int VPC_, int KT_>
struct LongLine {
    using G = G_;
    using T = typename G::T;
    static constexpr int N = G::N0, H = (N - 1) / 2, KT = KT_, VPC = VPC_;
    static_assert(x_direct_sum(N), "prime x lines above 31 points");
    static constexpr int LINES = VPC * G::N1 * G::N2;
    static constexpr int GROUPS = (H + KT - 1) / KT;
    static constexpr int TASKS = LINES * GROUPS;  // task t: line t % LINES, outputs of group t / LINES

    struct Acc {
        double are[KT], aim[KT], bre[KT], bim[KT];
        double sre, sim;  // output 0
    };

    FFT_HD static int slot(int l, int x)
    {
        const int z = l % G::N2, t = l / G::N2;
        return G::off((t / G::N1 * N + x) * G::N1 + t % G::N1, z);
    }

    // `tw[e]` = {cos, sin}(2 pi e / N)
    FFT_HD static void sums(const cx<T> *sm, const cx<double> *tw, int t, Acc &a)
    {
        const int l = t % LINES, k0 = t / LINES * KT + 1;
        constexpr int STEP = G::N1 * G::P2;  // x -> x + 1 (row pitch layouts)
        static_assert(G::POL != 2, "row pitch layouts");
        const cx<T> *p = sm + slot(l, 0);
        a.sre = (double)p[0].re;
        a.sim = (double)p[0].im;
        int e[KT];
#pragma unroll
        for (int i = 0; i < KT; ++i) {
            a.are[i] = a.sre;
            a.aim[i] = a.sim;
            a.bre[i] = a.bim[i] = 0.0;
            e[i] = 0;
        }
        for (int j = 1; j <= H; ++j) {
            const cx<T> f = p[j * STEP], b = p[(N - j) * STEP];
            const double ur = (double)f.re + (double)b.re, ui = (double)f.im + (double)b.im;
            const double wr = (double)f.re - (double)b.re, wi = (double)f.im - (double)b.im;
            a.sre += ur;
            a.sim += ui;
#pragma unroll
            for (int i = 0; i < KT; ++i) {
                e[i] += k0 + i;
                if (e[i] >= N) e[i] -= N;
                const cx<double> w = tw[e[i]];
                a.are[i] += ur * w.re;
                a.aim[i] += ui * w.re;
                a.bre[i] += wr * w.im;
                a.bim[i] += wi * w.im;
            }
        }
    }

    // The task's outputs into the line's slots, scaled for the inverse, once
    // every task of the group of volumes has its sums.
    template <int S>
    FFT_HD static void put(cx<T> *sm, int t, const Acc &a, T scale)
    {
        const int l = t % LINES, g = t / LINES;
        auto at = [&](int k, double re, double im) {
            cx<T> r = {(T)re, (T)im};
            if constexpr (S > 0) r = cscale(r, scale);
            sm[slot(l, k)] = r;
        };
        if (g == 0) at(0, a.sre, a.sim);
#pragma unroll
        for (int i = 0; i < KT; ++i) {
            const int k = g * KT + i + 1;
            if (k > H) continue;
            // i S b = S (-b.im, b.re)
            const double ir = S > 0 ? -a.bim[i] : a.bim[i], ii = S > 0 ? a.bre[i] : -a.bre[i];
            at(k, a.are[i] + ir, a.aim[i] + ii);
            at(N - k, a.are[i] - ir, a.aim[i] - ii);
        }
    }
};

}  // namespace fft3d
