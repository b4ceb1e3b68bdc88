// recycle_kernels.cu -- kernel family STREAM, RECYCLE variants: volumes of which
// an SM holds one (16x16x32, 23^3 and 24^3 complex double, 131-221 KB), with the
// next volume's rows loaded into shared memory as soon as the current one has
// read it.
//
// A second stage does not fit, so without this the SM's loads wait for its
// passes and its passes for the loads.  Here the x pass takes a chunk of y rows
// at a time, one line per thread, into registers; after a barrier the chunk's
// rows of all planes are free and the next volume's are loaded there by bulk
// copies while the chunk's lines are transformed and stored, the remaining
// chunks follow, and the next z pass starts on the first chunk.  Shared memory
// beyond one volume holds further planes of the next one (recycle.cuh).
//
// Measured over 96 MB (floor 30 us at 6.65 TB/s), the best kernel before and this
// one: 16x16x32 c128 60.9 (directp) / 51.1 us, 27 planes in the ring (16 planes:
// 53.0); 24^3 c128 78.3 (VOLUME) / 59.5; 30^3 c64 85.2 (VOLUME) / 61.8; 16^3 c128,
// three CTAs an SM, 44.9 (STREAM) / 43.0; 23^3 c128 88.6 (VOLUME) / 84.8, bound by
// the FP64 operations of its 23-point lines (66 us for 1024 volumes at the pipe's
// full rate, 147 us measured).  Chunks of one line per thread on twice the threads
// were slower (24^3: 72.5 us; 23^3: 112-138 us): their registers spill.  17^3, two
// CTAs an SM, takes 62 us against 43.5 us for the two-stage STREAM kernel.
#include "internal.h"
#include "ptx.cuh"
#include "recycle.cuh"

namespace fft3d {

template <class RG, int S, int ALG, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_recycle(const cx<typename RG::T> *__restrict__ in, cx<typename RG::T> *__restrict__ out, long long nvol,
              typename RG::T scale, int *err)
{
    pdl_begin();
    using T = typename RG::T;
    using G = typename RG::G;
    constexpr int N0 = G::N0, N1 = G::N1, N2 = G::N2, NP = RG::NP, C = RG::C;
    static_assert((long long)G::V * G::EB % 16 == 0, "volumes stay aligned");
    static_assert(RG::RC * N2 <= NT, "one x line of a chunk per thread");
    extern __shared__ __align__(128) unsigned char smraw[];
    cx<T> *sm = reinterpret_cast<cx<T> *>(smraw);
    uint64_t *full = reinterpret_cast<uint64_t *>(smraw + RG::RING_BYTES);  // [slot][chunk]
    __shared__ int s_abort;
    const int tid = threadIdx.x;
    const long long mine = (nvol - blockIdx.x + gridDim.x - 1) / gridDim.x;  // this CTA's volumes
    const uint64_t pol_first = l2_policy_evict_first();
    // V and the rows are multiples of 16 bytes.  Complex float off a 16-byte boundary: the
    // threads copy by elements, asynchronously too, and each arrives on a chunk's barrier (233
    // volumes of 30^3: 44.4 us; 77.0 when one thread copied a chunk, VOLUME 45.3; aligned 34.5).
    const bool aligned = G::EB == 16 || (uintptr_t)in % 16 == 0;
    for (int i = tid; i < NP * C; i += NT) mbar_init(&full[i], aligned ? 1 : NT);
    if (tid == 0) s_abort = 0;
    fence_mbar_init();
    __syncthreads();

    // Row yy of chunk c of running plane q: its copy, and with row 0 the chunk's
    // byte count.
    auto issue_row = [&](unsigned q, int c, int yy) {
        const long long k = q / N0;
        if (k >= mine) return;
        const int x = (int)(q % N0), s = (int)(q % NP), y = c * RG::RC + yy;
        uint64_t *bar = &full[s * C + c];
        const uint32_t rows = (uint32_t)RG::rows(c);
        const cx<T> *src = in + (blockIdx.x + k * gridDim.x) * G::V + (x * N1 + y) * N2;
        if (yy == 0) mbar_arrive_expect_tx(bar, rows * RG::ROW_BYTES);
        if constexpr (G::P2 == N2) {  // the chunk's rows are one range
            if (yy == 0) bulk_g2s_hint(sm + G::off(s * N1 + y, 0), src, rows * RG::ROW_BYTES, bar, pol_first);
        } else {
            bulk_g2s_hint(sm + G::off(s * N1 + y, 0), src, RG::ROW_BYTES, bar, pol_first);
        }
    };
    // Chunk c of the running planes [q, q + planes), by all threads.
    auto issue = [&](unsigned q, int planes, int c) {
        if constexpr (G::EB == 8) {
            if (!aligned) {
                for (unsigned p = q; p < q + planes && p / N0 < mine; ++p) {
                    const int x = (int)(p % N0), s = (int)(p % NP), y = c * RG::RC;
                    const cx<T> *src = in + (blockIdx.x + p / N0 * (long long)gridDim.x) * G::V + (x * N1 + y) * N2;
                    for (int j = tid; j < RG::rows(c) * N2; j += NT)
                        cp_async_8(sm + G::off(s * N1 + y + j / N2, j % N2), src + j);
                    cp_async_mbar_arrive_noinc(&full[s * C + c]);
                }
                return;
            }
        }
        for (int i = tid; i < planes * RG::rows(c); i += NT) issue_row(q + i / RG::rows(c), c, i % RG::rows(c));
    };
#pragma unroll
    for (int c = 0; c < C; ++c) issue(0u, NP, c);

    unsigned q0 = 0;  // running number of the current volume's plane 0
    int base = 0;     // its slot
    for (long long k = 0; k < mine; ++k, q0 += N0) {
        for (int t = tid; t < G::ROWS; t += NT) {
            int x, y, c;
            RG::z_row(t, &x, &y, &c);
            const int s = RG::slot(base, x);
            if (!mbar_wait_bounded(&full[s * C + c], ((q0 + x) / NP) & 1)) s_abort = 1;
            pass_z<G, S, ALG>(sm, s * N1 + y);
        }
        __syncthreads();
        if (s_abort) break;
        for (int l = tid; l < N0 * N2; l += NT)
            pass_y<G, S, ALG>(sm, RG::slot(base, l / N2) * N2 + l % N2);
        __syncthreads();
        cx<T> *gout = out + (blockIdx.x + k * gridDim.x) * G::V;
#pragma unroll 1
        for (int c = 0; c < C; ++c) {
            const bool line = tid < RG::rows(c) * N2;
            cx<T> v[N0];
            if (line) RG::x_load(sm, base, c, tid, v);
            fence_proxy_async_smem();  // these reads before the copies into the same rows
            __syncthreads();
            issue(q0 + NP, N0, c);
            if (line) RG::template x_store<S, ALG>(gout, c, tid, v, scale);
        }
        base = RG::slot(base, N0 % NP);
    }

    if (s_abort) {
        if (tid == 0) {
            report_error(err, DEV_ERR_LOAD_TIMEOUT);
            // bounded wait for every load in flight: planes q0 .. q0 + NP - 1
            for (unsigned q = q0; q < q0 + NP; ++q)
                for (int c = 0; c < C; ++c)
                    if (q / N0 < mine) mbar_wait_bounded(&full[q % NP * C + c], (q / NP) & 1);
        }
        __syncthreads();
    }
}

template <int N0, int N1, int N2, typename T, int PITCH, int NP, int RC, int S, int ALG, int NT, int MINB>
static void add_recycle(std::vector<KernelEntry> &out, const char *name)
{
    using RG = Recycle<N0, N1, N2, T, PITCH, NP, RC>;
    KernelEntry e;
    e.n0 = N0;
    e.n1 = N1;
    e.n2 = N2;
    e.precision = sizeof(T) == 8 ? FFT3D_B200_C128 : FFT3D_B200_C64;
    e.sign = S;
    e.family = FAM_STREAM;  // persistent launch over volumes: (in, out, nvol, scale, err)
    e.alg = ALG;
    e.vpc = 1;
    e.threads = NT;
    e.smem = RG::SMEM_BYTES;
    e.func = (const void *)&k_recycle<RG, S, ALG, NT, MINB>;
    e.name = name;
    out.push_back(e);
}

#define FFT3D_RECYCLE(N0, N1, N2, T, ALG, PITCH, NP, RC, NT, MINB)                                 \
    add_recycle<N0, N1, N2, T, PITCH, NP, RC, -1, ALG, NT, MINB>(                                  \
        out, "recycle " #N0 "x" #N1 "x" #N2 " " #T " alg" #ALG " np" #NP " rc" #RC " nt" #NT " minb" #MINB); \
    add_recycle<N0, N1, N2, T, PITCH, NP, RC, +1, ALG, NT, MINB>(                                  \
        out, "recycle " #N0 "x" #N1 "x" #N2 " " #T " alg" #ALG " np" #NP " rc" #RC " nt" #NT " minb" #MINB)

void register_recycle_kernels(std::vector<KernelEntry> &out)
{
    // 384 volumes 51.1 us; DIRECT, pipelined and plain, 60.9 and 73.2 (10.3 against 9.4 us for
    // one volume, where VOLUME takes 8.2): not compiled for this extent any more
    FFT3D_RECYCLE(16, 16, 32, double, 0, 33, 27, 8, 256, 1);
    FFT3D_RECYCLE(23, 23, 23, double, 0, 23, 23, 12, 288, 1);
    FFT3D_RECYCLE(24, 24, 24, double, 0, 25, 24, 8, 192, 1);
    FFT3D_RECYCLE(16, 16, 16, double, 0, 17, 16, 8, 128, 3);
    FFT3D_RECYCLE(30, 30, 30, float, 0, 30, 30, 10, 320, 1);
}

}  // namespace fft3d
