// recycle.cuh -- index arithmetic of the RECYCLE kernels (host and device): one
// volume per CTA in a ring of NP >= N0 plane slots, its y rows cut into chunks of
// RC, each chunk of a plane loaded on its own.
//
// Plane x of the CTA's k-th volume has the running number q = k N0 + x and lives
// in slot q mod NP.  The x pass of a chunk reads the chunk's rows of every plane
// for the last time; they are then free for planes q + NP.
#pragma once

#include "volume.cuh"

namespace fft3d {

template <int N0, int N1, int N2, typename T_, int PITCH, int NP_, int RC_>
struct Recycle {
    using T = T_;
    using G = Geom<N0, N1, N2, T, PITCH>;
    static constexpr int NP = NP_, RC = RC_, C = (N1 + RC - 1) / RC;
    static_assert(NP >= N0 && PITCH >= N2 && RC >= 1 && RC <= N1, "whole volumes in the ring");
    static constexpr int ROW_BYTES = N2 * G::EB;
    static_assert(ROW_BYTES % 16 == 0 && (PITCH * G::EB) % 16 == 0, "bulk row copies: 16-byte rows");
    static constexpr int RING_BYTES = (NP * N1 * PITCH * G::EB + 127) / 128 * 128;
    static constexpr int SMEM_BYTES = RING_BYTES + 8 * NP * C;

    FFT_HD static constexpr int rows(int c) { return c * RC + RC <= N1 ? RC : N1 - c * RC; }
    // slot of plane x of a volume whose plane 0 is in slot `base`
    FFT_HD static int slot(int base, int x)
    {
        if constexpr (NP == N0) return x;
        const int s = base + x;
        return s >= NP ? s - NP : s;
    }
    // z-pass task t -> row (x, y), chunk by chunk
    FFT_HD static void z_row(int t, int *x, int *y, int *c)
    {
        const int cc = t / (N0 * RC);
        const int rem = t - cc * (N0 * RC);
        const int n = rows(cc);
        *c = cc;
        *x = rem / n;
        *y = cc * RC + rem % n;
    }
    // x line `l` of chunk c into registers; and out, scaled for the inverse
    FFT_HD static void x_load(const cx<T> *sm, int base, int c, int l, cx<T> (&v)[N0])
    {
        const int y = c * RC + l / N2, z = l % N2;
#pragma unroll
        for (int j = 0; j < N0; ++j) v[j] = sm[G::off(slot(base, j) * N1 + y, z)];
    }
    template <int S, int ALG>
    FFT_HD static void x_store(cx<T> *gout, int c, int l, cx<T> (&v)[N0], T scale)
    {
        cx<T> *o = gout + c * RC * N2 + l;
        dft_emit<N0, S, T, ALG>(v, [&](int j, cx<T> r) {
            if constexpr (S > 0) r = cscale(r, scale);
            o[j * (N1 * N2)] = r;
        });
    }
};

}  // namespace fft3d
