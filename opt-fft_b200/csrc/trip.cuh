// trip.cuh -- work decomposition of the TRIP kernel (host and device): cubes N^3
// beyond one SM's shared memory, N = A x B, transformed in plane and row items
// (twopass.cuh) whose threads hold at most max(A, B^2) points.
//
// A whole N-point complex-double line in one thread needs 4N registers, and split
// into two stages of 8 points a line crosses shared memory four times.  Here a
// plane of N x N points takes three trips through the registers, with A, B^2 and A
// points a task:
//   trip 1  z, A-point DFTs over z = B a + b (class b): HBM -> shared memory;
//           lanes run along b first, so a warp reads runs of B points of a row;
//   trip 2  the B-point half of z and the B-point half of y together;
//   trip 3  y, A-point DFTs; lanes along z: shared memory -> scratch ring.
// and a row item (G y-rows of every x-plane) two: A-point DFTs along x straight
// from the ring, B-point DFTs straight to the output, lanes along z in both.  Every
// axis is split by Cooley-Tukey (the mixed-radix route of the reference's
// python/fft3d.py:166-188), with the twiddles between its halves in trip 2 and in
// the second stage of a row item.
//
// Shared memory of a plane item: y = A m1 + m2 of plane g at (g N + y) P, point
// (ka, b) of its row at b ZB + ka, so z = ka + A kb comes to lie at kb ZB + ka.  For
// 64 = 16 x 4, ZB = 17 and P = 68 let every 128-byte phase of the three trips meet
// distinct banks, in both precisions.
#pragma once

#include "codelets.cuh"
#include "volume.cuh"

namespace fft3d {

template <int N>
struct TripSplit;
template <>
struct TripSplit<64> {
    static constexpr int A = 16, B = 4, ZB = 17, P = 68;
};

template <int N_, typename T_, int G_>
struct Trip {
    using T = T_;
    using L = TripSplit<N_>;
    static constexpr int N = N_, G = G_, A = L::A, B = L::B, ZB = L::ZB, P = L::P;
    static_assert(A * B == N && N % G == 0, "N = A x B, whole items");
    static constexpr long long PLANE = (long long)N * N;
    static constexpr int COLS = G * N;              // columns (y, z) of a row item
    static constexpr int T1 = G * N * B, T2 = G * A * A, T3 = G * B * N;  // tasks of a plane item
    static constexpr int R1 = COLS * B, R2 = COLS * A;                    // tasks of a row item
    static constexpr int PLANE_SM = G * N * P, ROW_SM = N * COLS;
    static constexpr int SM_ELEMS = PLANE_SM > ROW_SM ? PLANE_SM : ROW_SM;
    static constexpr int TW = (B - 1) * A;          // twiddle table entries

    // entry (b, ka), b >= 1: {cos, sin}(2 pi b ka / N)
    FFT_HD static constexpr int tw_slot(int b, int ka) { return (b - 1) * A + ka; }
    FFT_HD static cx<T> tw_entry(int e)
    {
        const auto w = Tab<T>::tw(tw_off(N) + (e / A + 1) * (e % A));  // (b ka) < N
        return {w.x, w.y};
    }
    template <int S>
    FFT_HD static cx<T> mul_tw(cx<T> v, cx<T> w)
    {
        const T s = S > 0 ? w.im : -w.im;
        return {v.re * w.re - v.im * s, v.re * s + v.im * w.re};
    }

    // trip 1, its loads and the rest; `in` is the item's first plane
    template <class Load>
    FFT_HD static void trip1_load(const cx<T> *in, int t, cx<T> (&v)[A], Load load)
    {
        const cx<T> *src = in + t / B * N + t % B;
#pragma unroll
        for (int a = 0; a < A; ++a) v[a] = load(src + B * a);
    }
    template <int S>
    FFT_HD static void trip1_store(cx<T> *sm, int t, cx<T> (&v)[A])
    {
        dft<A, S, T>(v);
        cx<T> *d = sm + t / B * P + t % B * ZB;
#pragma unroll
        for (int a = 0; a < A; ++a) d[a] = v[a];
    }

    // trip 2, in place: B x B points of one (ka, m2)
    template <int S>
    FFT_HD static void trip2(cx<T> *sm, const cx<T> *tw, int t)
    {
        const int ka = t % A, q = t / A;
        const int m2 = q % A, g = q / A;
        cx<T> *d = sm + (g * N + m2) * P + ka;
        cx<T> v[B][B];  // [m1][b]
#pragma unroll
        for (int b = 0; b < B; ++b)
#pragma unroll
            for (int m1 = 0; m1 < B; ++m1) v[m1][b] = d[m1 * (A * P) + b * ZB];
#pragma unroll
        for (int b = 1; b < B; ++b) {
            const cx<T> w = tw[tw_slot(b, ka)];
#pragma unroll
            for (int m1 = 0; m1 < B; ++m1) v[m1][b] = mul_tw<S>(v[m1][b], w);
        }
#pragma unroll
        for (int m1 = 0; m1 < B; ++m1) dft<B, S, T>(v[m1]);
#pragma unroll
        for (int kb = 0; kb < B; ++kb) {
            cx<T> c[B];
#pragma unroll
            for (int m1 = 0; m1 < B; ++m1) c[m1] = v[m1][kb];
            dft<B, S, T>(c);
#pragma unroll
            for (int l1 = 0; l1 < B; ++l1) v[l1][kb] = c[l1];
        }
#pragma unroll
        for (int l1 = 1; l1 < B; ++l1) {
            const cx<T> w = tw[tw_slot(l1, m2)];
#pragma unroll
            for (int kb = 0; kb < B; ++kb) v[l1][kb] = mul_tw<S>(v[l1][kb], w);
        }
#pragma unroll
        for (int l1 = 0; l1 < B; ++l1)
#pragma unroll
            for (int kb = 0; kb < B; ++kb) d[l1 * (A * P) + kb * ZB] = v[l1][kb];
    }

    // trip 3: `dst` is the item's first plane in the scratch slot
    template <int S, class Store>
    FFT_HD static void trip3(const cx<T> *sm, cx<T> *dst, int t, Store store)
    {
        const int z = t % N, q = t / N;
        const int l1 = q % B, g = q / B;
        const cx<T> *s = sm + (g * N + l1 * A) * P + (z / A) * ZB + z % A;
        cx<T> v[A];
#pragma unroll
        for (int m2 = 0; m2 < A; ++m2) v[m2] = s[m2 * P];
        dft<A, S, T>(v);
        cx<T> *o = dst + (long long)g * PLANE + z;
#pragma unroll
        for (int l2 = 0; l2 < A; ++l2) store(o + (l1 + B * l2) * N, v[l2]);
    }

    // row item, first stage; `src` is the first y-row of the item in the slot
    template <class Load>
    FFT_HD static void row1_load(const cx<T> *src, int t, cx<T> (&v)[A], Load load)
    {
        const int c = t % COLS, b = t / COLS;
#pragma unroll
        for (int a = 0; a < A; ++a) v[a] = load(src + (B * a + b) * PLANE + c);
    }
    template <int S>
    FFT_HD static void row1_store(cx<T> *sm, int t, cx<T> (&v)[A])
    {
        const int c = t % COLS, b = t / COLS;
        dft<A, S, T>(v);
        cx<T> *d = sm + b * (A * COLS) + c;
#pragma unroll
        for (int ka = 0; ka < A; ++ka) d[ka * COLS] = v[ka];
    }

    // row item, second stage: `dst` is the first y-row of the item in the output
    template <int S, class Store>
    FFT_HD static void row2(const cx<T> *sm, const cx<T> *tw, cx<T> *dst, int t, T scale, Store store)
    {
        const int c = t % COLS, ka = t / COLS;
        cx<T> v[B];
#pragma unroll
        for (int b = 0; b < B; ++b) v[b] = sm[(b * A + ka) * COLS + c];
#pragma unroll
        for (int b = 1; b < B; ++b) v[b] = mul_tw<S>(v[b], tw[tw_slot(b, ka)]);
        dft<B, S, T>(v);
#pragma unroll
        for (int kb = 0; kb < B; ++kb) {
            cx<T> r = v[kb];
            if constexpr (S > 0) r = cscale(r, scale);
            store(dst + (ka + A * kb) * PLANE + c, r);
        }
    }
};

}  // namespace fft3d
