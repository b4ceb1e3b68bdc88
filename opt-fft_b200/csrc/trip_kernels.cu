// trip_kernels.cu -- kernel family TWOPASS, TRIP variants: plane and row items
// through the L2-resident scratch ring (twopass.cuh), every line split over
// several tasks (trip.cuh).
//
// Control is a warp of its own.  Its first thread takes tickets, polls the
// counters that an item depends on while the worker warps transform the item
// before it, and publishes finished items, so no worker waits out the L2 round
// trips of a ticket, an acquire or a release.  Items pass through a two-entry
// mailbox with one mbarrier each way.  An item that is posted has all it depends
// on, and the items a CTA holds are polled and published independently of each
// other, so the ticket-order argument against deadlock (twopass.cuh) holds.  A
// slot is published by one cumulative gpu-scope release after every worker
// arrived on the item's mbarrier.
//
// Input, ring and output move between HBM or L2 and the registers without a
// staging copy; the first loads of an item are issued before the barrier that
// frees shared memory.
#include "internal.h"
#include "ptx.cuh"
#include "trip.cuh"
#include "twopass.cuh"
#include "twopass_dev.cuh"

namespace fft3d {

// Item of the mailbox: a ticket, or why there are no more.
constexpr long long TRIP_END = -1;    // every ticket is taken
constexpr long long TRIP_ABORT = -2;  // a wait ran out, here or in another CTA

// The control thread: returns false when a wait ran out.
template <class TG>
__device__ __forceinline__ bool trip_control(TwoPassCtl *ctl, long long nvol, int R, int D,
                                             volatile long long *mail, uint64_t *full, uint64_t *done)
{
    const long long total = (long long)(TG::NA + TG::NB) * nvol;
    long long t = (long long)atomicAdd(&ctl->ticket, 1ull);
    unsigned posted = 0, freed = 0;  // items handed to the workers, and published
    unsigned *publish = nullptr, *publish_next = nullptr;  // the counters of the oldest item and of the one after it
    unsigned long long since = globaltimer_ns();  // the last step forward
    auto post = [&](long long item) {
        mail[posted & 1] = item;
        mbar_arrive(&full[posted & 1]);
    };
    for (;;) {
        // test_wait: try_wait may suspend the thread for as long as the item takes, and
        // the next item's counter would be polled only then
        if (freed != posted && mbar_test_wait(&done[freed & 1], (freed >> 1) & 1)) {
            red_release_gpu_add(publish, 1u);
            publish = publish_next;
            ++freed;
            since = globaltimer_ns();
        }
        const bool late = globaltimer_ns() - since > kCounterWaitNs;
        if (posted - freed == 2 || (t >= total && freed != posted)) {  // the workers are on it
            if (late) return false;
            continue;
        }
        if (t >= total) {
            post(TRIP_END);
            return true;
        }
        const TwoPassItem it = twopass_decode(t, nvol, TG::NA, TG::NB, D);
        const int slot = (int)(it.vol % R);
        const unsigned round = (unsigned)(it.vol / R);
        // a plane item's slot must have been read out, a row item's planes be there
        unsigned *planes = &ctl->cnt[slot], *rows = &ctl->cnt[TWOPASS_RMAX + slot];
        const unsigned target = it.plane ? (unsigned)TG::NB * round : (unsigned)TG::NA * (round + 1u);
        if (target == 0 || ld_acquire_gpu(it.plane ? rows : planes) >= target) {
            (posted == freed ? publish : publish_next) = it.plane ? planes : rows;
            post(t);
            ++posted;
            t = (long long)atomicAdd(&ctl->ticket, 1ull);
            since = globaltimer_ns();
        } else {
            if (late || ld_acquire_gpu(&ctl->abort) != 0) {
                post(TRIP_ABORT);
                return false;
            }
            __nanosleep(64);
        }
    }
}

template <int N, typename T, int S, int G, int NT, int MINB>
__global__ void __launch_bounds__(NT + 32, MINB)
    k_trip(const cx<T> *__restrict__ in, cx<T> *__restrict__ out, long long nvol, T scale, int *err,
           unsigned char *work, int R, int D)
{
    pdl_begin();
    using TR = Trip<N, T, G>;
    using TG = TwoPassGeom<N, N, N, T, G>;
    static_assert(NT % 32 == 0, "whole worker warps");
    extern __shared__ __align__(128) unsigned char smraw[];
    cx<T> *sm = reinterpret_cast<cx<T> *>(smraw);
    __shared__ cx<T> s_tw[TR::TW];
    __shared__ long long s_mail[2];
    __shared__ __align__(8) uint64_t s_full[2], s_done[2];
    TwoPassCtl *ctl = reinterpret_cast<TwoPassCtl *>(work);
    cx<T> *ring = reinterpret_cast<cx<T> *>(work + TWOPASS_CTL_BYTES);
    const int tid = threadIdx.x;
    for (int e = tid; e < TR::TW; e += NT + 32) s_tw[e] = TR::tw_entry(e);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_done[i], NT);
        }
    }
    __syncthreads();

    if (tid >= NT) {
        if (tid == NT && !trip_control<TG>(ctl, nvol, R, D, s_mail, s_full, s_done)) {
            report_error(err, DEV_ERR_DEP_TIMEOUT);
            atomicExch(&ctl->abort, 1u);
        }
    } else {
        const uint64_t pol_first = l2_policy_evict_first();
        const uint64_t pol_last = l2_policy_evict_last();
        auto ld_in = [&](const cx<T> *p) { return ld_hint(p, pol_first); };
        auto ld_ring = [&](const cx<T> *p) { return load_l2(p); };
        auto st_ring = [&](cx<T> *p, cx<T> v) { st_hint(p, v, pol_last); };
        auto st_out = [&](cx<T> *p, cx<T> v) { store_out(p, v); };
        for (unsigned k = 0;; ++k) {
            // The workers leave together, by a vote at an item's first barrier: one whose
            // wait ran out while another's was still answered must not be missing at
            // the barriers that follow.
            const bool posted = mbar_wait_timed(&s_full[k & 1], (k >> 1) & 1);
            const long long ticket = *(volatile long long *)&s_mail[k & 1];
            if (!posted || ticket < 0) {
                if (!posted) report_error(err, DEV_ERR_QUEUE_TIMEOUT);
                named_barrier_any(1, NT, true);
                break;
            }
            const TwoPassItem it = twopass_decode(ticket, nvol, TG::NA, TG::NB, D);
            cx<T> *sv = ring + it.vol % R * TG::V;
            cx<T> v[TR::A];
            if (it.plane) {
                const long long p0 = (long long)it.j * G * TR::PLANE;
                const cx<T> *src = in + it.vol * TG::V + p0;
                if (tid < TR::T1) TR::trip1_load(src, tid, v, ld_in);
                if (named_barrier_any(1, NT, false)) break;  // the item before has left shared memory
                if (tid < TR::T1) TR::template trip1_store<S>(sm, tid, v);
                for (int t = tid + NT; t < TR::T1; t += NT) {
                    TR::trip1_load(src, t, v, ld_in);
                    TR::template trip1_store<S>(sm, t, v);
                }
                named_barrier_sync(1, NT);
                for (int t = tid; t < TR::T2; t += NT) TR::template trip2<S>(sm, s_tw, t);
                named_barrier_sync(1, NT);
                for (int t = tid; t < TR::T3; t += NT) TR::template trip3<S>(sm, sv + p0, t, st_ring);
            } else {
                const long long r0 = (long long)it.j * G * N;
                if (tid < TR::R1) TR::row1_load(sv + r0, tid, v, ld_ring);
                if (named_barrier_any(1, NT, false)) break;
                if (tid < TR::R1) TR::template row1_store<S>(sm, tid, v);
                for (int t = tid + NT; t < TR::R1; t += NT) {
                    TR::row1_load(sv + r0, t, v, ld_ring);
                    TR::template row1_store<S>(sm, t, v);
                }
                named_barrier_sync(1, NT);
                // every load of the slot has returned: drop its lines from L2 unwritten
                twopass_discard_rows<TG>(sv, it.j, tid, NT);
                cx<T> *dst = out + it.vol * TG::V + r0;
                for (int t = tid; t < TR::R2; t += NT) TR::template row2<S>(sm, s_tw, dst, t, scale, st_out);
            }
            mbar_arrive(&s_done[k & 1]);
        }
    }
    __syncthreads();
    twopass_leave(ctl, tid);
}

template <int N, typename T, int S, int G, int NT, int MINB>
static void add_trip(std::vector<KernelEntry> &out, const char *name)
{
    KernelEntry e;
    e.n0 = e.n1 = e.n2 = N;
    e.precision = sizeof(T) == 8 ? FFT3D_B200_C128 : FFT3D_B200_C64;
    e.sign = S;
    e.family = FAM_TWOPASS;  // same launch arguments and workspace as k_twopass
    e.alg = 2048;
    e.vpc = G;
    e.threads = NT + 32;  // and the control warp
    e.smem = Trip<N, T, G>::SM_ELEMS * (int)sizeof(cx<T>);
    e.func = (const void *)&k_trip<N, T, S, G, NT, MINB>;
    e.name = name;
    out.push_back(e);
}

#define FFT3D_TRIP(N, T, G, NT, MINB)                                                             \
    add_trip<N, T, -1, G, NT, MINB>(out, "twopass " #N "x" #N "x" #N " " #T " g" #G " trip nt" #NT \
                                         " minb" #MINB);                                          \
    add_trip<N, T, +1, G, NT, MINB>(out, "twopass " #N "x" #N "x" #N " " #T " g" #G " trip nt" #NT \
                                         " minb" #MINB)

// Measured over 96 MB (floor 30 us at 6.65 TB/s), the staged kernel (two 8-point
// stages a line through shared memory, twopass_kernels.cu) and this one: 64^3 c128
// 92.7 / 74.0 us.  Movement through the ring alone, without the trips through
// shared memory or any wait, takes 45 us, the trips add 13 us and the arithmetic
// 6 us.  Two CTAs of 256 workers an SM; three spill (100 us).  The same split as
// 9 x 4 for 36^3 takes 74-79 us against 70 us for one line a thread (bulkqh), 8 x 3
// for 24^3 86 us against 78 us, 10 x 3 for 30^3 and 9 x 5 for 45^3 as long as their
// one-line kernels, and 16 x 4 in complex float 79.5 us against 81.0 us: not kept.
void register_trip_kernels(std::vector<KernelEntry> &out)
{
    FFT3D_TRIP(64, double, 1, 256, 2);
}

}  // namespace fft3d
