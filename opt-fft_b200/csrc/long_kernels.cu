// long_kernels.cu -- kernel family VOLUME, LONG variants: volumes with prime x
// lines of 47, 83 or 97 points (longline.cuh).
//
// One CTA per group of volumes: staging, z and y passes as k_volume; the x lines
// are then summed by several threads each, put back in place and copied out in
// order.  The VOLUME kernel gives a line to one thread, which reads a factor from
// global memory for each of its N^2 products; with a few lines a volume an SM
// runs a few dozen such threads.  What bounds this one is the FP64 pipe: 4 H^2
// multiply-adds a line, 17 us for 48 MB of 97x2x1 complex double at its full rate
// and 33 us for complex float (twice the lines, sums in double as before).
// Measured over 48 MB, VOLUME and LONG: complex double 97x2x1 1325 / 57 us, 83x2x1
// 970 / 57, 47x3x2 175 / 52; complex float 1672 / 99, 1076 / 97, 248 / 75.  More
// outputs a task read shared memory less often but leave fewer warps: 4 to 8 were
// tried with 160-384 threads (97x2x1 c128: 4 60 us, 6 57 us, 8 93 us).
#include "internal.h"
#include "longline.cuh"
#include "ptx.cuh"

namespace fft3d {

template <class LL, int S, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_long(const cx<typename LL::T> *__restrict__ in, cx<typename LL::T> *__restrict__ out, long long nvol,
           typename LL::T scale)
{
    pdl_begin();
    using T = typename LL::T;
    using G = typename LL::G;
    constexpr int VPC = LL::VPC;
    static_assert(LL::TASKS <= NT, "one x-line task per thread");
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *sm = reinterpret_cast<cx<T> *>(smraw);
    __shared__ cx<double> s_tw[LL::N];
    const int tid = threadIdx.x;
    const long long v0 = (long long)blockIdx.x * VPC;
    const int nv = nvol - v0 < VPC ? (int)(nvol - v0) : VPC;
    const cx<T> *gin = in + v0 * G::V;
    cx<T> *gout = out + v0 * G::V;

    for (int e = tid; e < LL::N; e += NT) {
        const auto w = line_tw<LL::N, double>(e);
        s_tw[e] = {w.x, w.y};
    }
    for (int g = tid; g < nv * G::V; g += NT) stage_in<G>(sm, gin, g);
    __syncthreads();
    if constexpr (G::N2 > 1) {
        for (int r = tid; r < nv * G::ROWS; r += NT) pass_z<G, S, ALG_DEFAULT>(sm, r);
        __syncthreads();
    }
    if constexpr (G::N1 > 1) {
        for (int l = tid; l < nv * G::N0 * G::N2; l += NT) pass_y<G, S, ALG_DEFAULT>(sm, l);
        __syncthreads();
    }
    const bool task = tid < LL::TASKS && tid % LL::LINES < nv * G::N1 * G::N2;
    typename LL::Acc a;
    if (task) LL::sums(sm, s_tw, tid, a);
    __syncthreads();
    if (task) LL::template put<S>(sm, tid, a, scale);
    __syncthreads();
    for (int g = tid; g < nv * G::V; g += NT) store_out(gout + g, sm[G::off(g / G::N2, g % G::N2)]);
}

template <int N0, int N1, int N2, typename T, int S, int VPC, int KT, int NT, int MINB>
static void add_long(std::vector<KernelEntry> &out, const char *name)
{
    using G = Geom<N0, N1, N2, T>;
    KernelEntry e;
    e.n0 = N0;
    e.n1 = N1;
    e.n2 = N2;
    e.precision = sizeof(T) == 8 ? FFT3D_B200_C128 : FFT3D_B200_C64;
    e.sign = S;
    e.family = FAM_VOLUME;
    e.alg = 0;
    e.vpc = VPC;
    e.threads = NT;
    e.smem = VPC * G::PV * G::EB;
    e.func = (const void *)&k_long<LongLine<G, VPC, KT>, S, NT, MINB>;
    e.name = name;
    out.push_back(e);
}

#define FFT3D_LONG(N0, N1, N2, T, VPC, KT, NT, MINB)                                               \
    add_long<N0, N1, N2, T, -1, VPC, KT, NT, MINB>(                                                \
        out, "long " #N0 "x" #N1 "x" #N2 " " #T " vpc" #VPC " kt" #KT " nt" #NT " minb" #MINB);     \
    add_long<N0, N1, N2, T, +1, VPC, KT, NT, MINB>(                                                \
        out, "long " #N0 "x" #N1 "x" #N2 " " #T " vpc" #VPC " kt" #KT " nt" #NT " minb" #MINB)

void register_long_kernels(std::vector<KernelEntry> &out)
{
    FFT3D_LONG(97, 2, 1, double, 16, 6, 256, 2);
    FFT3D_LONG(83, 2, 1, double, 16, 6, 224, 2);
    FFT3D_LONG(47, 3, 2, double, 8, 8, 160, 3);
    FFT3D_LONG(97, 2, 1, float, 16, 4, 384, 2);
    FFT3D_LONG(83, 2, 1, float, 16, 7, 192, 3);
    FFT3D_LONG(47, 3, 2, float, 8, 8, 160, 3);
}

}  // namespace fft3d
