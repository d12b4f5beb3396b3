// Pieces shared by the solvers that keep one right-hand side's Krylov fields in
// the registers and shared memory of a thread-block cluster (eo_cluster.cu,
// cg_cluster.cu).
//
// CTAs of a cluster exchange halo rows and partial sums by asynchronous remote
// stores (st.async) that count their bytes on an mbarrier of the receiving CTA.
// A phase then waits only for the data it reads, and only in the threads that
// read it: no cluster barrier and no memory barrier in the iteration, where a
// cluster barrier per phase held every warp for the slowest CTA and its release
// flushed each warp's stores first.
//
// A receiver's barrier is used for one message at a time: the sender's next
// message into the same place needs data the receiver sends only after it has
// read the last one (each solver says why at its phases).
//
// A wait that runs past the limit is noted in the waiting lane (`bad`). The warps of
// a CTA may then hold different values of a sum, so each solver's loop is laid out
// such that warps on different ways meet at the same block barriers up to one that
// tells all of them (by __syncthreads_or of `bad`, or Quit). The CTA then gives up and
// goes to the next check point (Meet).
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace dwfb {
namespace cl {

namespace cg = cooperative_groups;

constexpr int kMaxCtas = 16;   // CTAs of a cluster
constexpr int kMaxWarps = 24;  // warps of a CTA

__device__ __forceinline__ unsigned smem_addr(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }

// Shared memory of this CTA at the same offset in CTA `rank` of the cluster, as
// a 32-bit address of the cluster's shared window.
__device__ __forceinline__ unsigned map(unsigned a, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

// Remote stores; their bytes count on the mbarrier `bar` of the same CTA.
__device__ __forceinline__ void send(unsigned a, float4 v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send(unsigned a, double v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void send(unsigned a, double2 v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)), "r"(bar)
                 : "memory");
}

// One arrival a phase; `missing` more that never come let no phase end (self test).
__device__ __forceinline__ void bar_init(unsigned bar, unsigned missing = 0)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(1u + missing) : "memory");
}
// The phase's one arrival, with the bytes it waits for (they may have begun to
// land before).
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait; false once it ran past the limit. The timer is read only now and
// then: a read takes about as long as a message.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, unsigned long long limit_ns)
{
    for (int n = 0; n < 256; ++n)
        if (bar_try(bar, parity))
            return true;
    const unsigned long long t0 = globaltimer_ns();
    for (unsigned n = 1; !bar_try(bar, parity); ++n)
        if (n % 256u == 0 && globaltimer_ns() - t0 > limit_ns)
            return false;
    return true;
}

// One lane's wait; a lane that is bad waits no more. ran_out() when it becomes bad.
template <typename F>
__device__ __forceinline__ void wait(unsigned bar, unsigned parity, unsigned long long limit_ns, int& bad, F ran_out)
{
    if (!bad && !bar_wait(bar, parity, limit_ns))
    {
        bad = 1;
        ran_out();
    }
}

// Cluster barrier (release / acquire at cluster scope).
__device__ __forceinline__ void sync() { cg::this_cluster().sync(); }

// The same after phases that write global memory (FP64 fields), with a
// device-scope fence ahead of the barrier.
__device__ __forceinline__ void sync_global()
{
    __threadfence();
    cg::this_cluster().sync();
}

// Sum over the cluster of one value per thread, in three steps: part() leaves
// every warp's sum in shared memory; after a block barrier send() (by one warp)
// adds them and sends the CTA's sum to every CTA's table; get() waits for the
// table and adds it up in a fixed order, the same bits in every warp of every
// CTA (unless the wait ran out: bad). One lane per warp polls: all threads polling,
// and a message per warp instead of per CTA, made the mbarrier the bottleneck (2.5 us
// a sum at 16 CTAs of 16 warps against 0.5). Thread 0 arms the slot's barrier in get(). A slot
// is sent again only after every warp of every CTA has sent something that it
// sends after its get() of that slot, and someone has waited for it.
struct Sum
{
    double* tab;   // [nslot][kMaxCtas], this CTA's
    double* wsum;  // [nslot][kMaxWarps]
    unsigned bar;  // mbarriers, 8 bytes apart
    int CS, rank;

    __device__ __forceinline__ void part(int slot, double v) const
    {
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0)
            wsum[slot * kMaxWarps + (threadIdx.x >> 5)] = v;
    }
    __device__ __forceinline__ void send(int slot) const
    {
        const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
        const double v = warp_sum(lane < nw ? wsum[slot * kMaxWarps + lane] : 0.0);
        if (lane < CS)
            cl::send(map(smem_addr(tab + slot * kMaxCtas + rank), lane), v, map(bar + 8u * slot, lane));
    }
    // Thread 0 arms no more once it is bad (its barrier may still be in the phase it
    // armed last).
    template <typename F>
    __device__ __forceinline__ double get(int slot, unsigned parity, unsigned long long limit_ns, int& bad,
                                          F ran_out) const
    {
        const int lane = threadIdx.x & 31;
        if (lane == 0 && !bad)
        {
            if (threadIdx.x == 0)
                bar_expect(bar + 8u * slot, unsigned(CS) * 8u);
            wait(bar + 8u * slot, parity, limit_ns, bad, ran_out);
        }
        __syncwarp();
        return warp_sum(lane < CS ? tab[slot * kMaxCtas + lane] : 0.0);
    }
};
// The solvers' fields begin at a multiple of 128 bytes behind the tables and
// barriers: a warp's 16-byte words then cover whole lines. FP64 CG at 24x20x10 / 32x32x8
// with 28 right-hand sides: 4.55 / 10.5 us an iteration there, 4.55 / 10.8 at 64 past
// it, 4.77 / 11.5 at 32, 5.02 / 11.5 to 12.4 at 16 and 80.
__host__ __device__ constexpr size_t head_bytes(size_t n) { return (n + 127) / 128 * 128; }

__host__ __device__ constexpr size_t sum_bytes(int nslot)
{
    return size_t(nslot) * (kMaxCtas + kMaxWarps) * sizeof(double);
}

// Check points: the cluster barriers at which the CTAs of a cluster agree on whether
// one of them gave up. Every CTA passes the same check points in the same order, and
// all leave at the first one that a CTA reached with `gave`, so no CTA stores into the
// shared memory of one that has left and none waits at a barrier that another will
// not reach. The barrier ends: a CTA gets there after at most two of its limited waits
// once another has stopped sending, and cluster barriers other than check points lie
// only where no CTA can give up since the last check point.
//
// A CTA that gives up writes the number of its next check point into every CTA's
// word; one that has passed its last check point may do so before a slower one
// has read its own word there, hence the number and not a flag. True: leave.
//
// The word and the count of check points passed lie in shared memory (8 bytes at
// `word`), and the even-odd solver looks at left() after its loop instead of leaving
// from within: a register or a way out of the loop more cost it spills and 1.5 %.
// Thread 0 counts after the barrier; a solver has a block barrier before its next
// check point.
struct Meet
{
    unsigned word;  // shared address

    __device__ __forceinline__ void init() const  // by one thread, before the first cluster barrier
    {
        asm volatile("st.shared::cta.v2.u32 [%0], {%1, %1};" ::"r"(word), "r"(0) : "memory");
    }
    __device__ __forceinline__ bool operator()(bool gave, int CS) const
    {
        unsigned n, v;
        asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(n) : "r"(word + 4u) : "memory");
        ++n;
        if (gave && int(threadIdx.x) < CS)
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map(word, int(threadIdx.x))), "r"(n) : "memory");
        sync_global();
        asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(word) : "memory");
        if (threadIdx.x == 0)
            asm volatile("st.shared::cta.u32 [%0], %1;" ::"r"(word + 4u), "r"(n) : "memory");
        return v == n;
    }
    // Whether the last check point said to leave (after a block barrier).
    __device__ __forceinline__ bool left() const
    {
        unsigned n, v;
        asm volatile("ld.volatile.shared::cta.v2.u32 {%0, %1}, [%2];" : "=r"(v), "=r"(n) : "r"(word) : "memory");
        return n != 0 && v == n;
    }
};

// The iteration from which a CTA gives up: one more than the iteration in which a
// wait ran out first (shared memory, zero: none has). All threads read it between the
// block barrier that starts an iteration and the next one; numbers noted meanwhile lie
// beyond the iteration, so all get the same answer however late they read. In the
// full-lattice CG 1.5 % faster (32x32 Wilson) than __syncthreads_or, whose result the
// barrier waits for.
struct Quit
{
    unsigned word;  // shared address

    __device__ __forceinline__ void init() const  // by one thread, before the first cluster barrier
    {
        asm volatile("st.shared::cta.u32 [%0], %1;" ::"r"(word), "r"(0) : "memory");
    }
    __device__ __forceinline__ void from(int it) const
    {
        unsigned old;
        asm volatile("atom.shared::cta.cas.b32 %0, [%1], 0, %2;" : "=r"(old) : "r"(word), "r"(it) : "memory");
    }
    __device__ __forceinline__ bool at(int it) const
    {
        unsigned v;
        asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(word) : "memory");
        return v - 1u < unsigned(it);
    }
};

constexpr int kGaveUp = -2;  // state of a right-hand side whose CTA gave up (beside RHS_ACTIVE and the status codes)

// After a check point that says to leave: all messages have been sent, those still on
// their way land long before this returns (they take about a microsecond).
__device__ __forceinline__ void settle()
{
    const unsigned long long t0 = globaltimer_ns();
    for (int i = 0; i < 100000 && globaltimer_ns() - t0 < 1000000ull; ++i)
        __nanosleep(1000);
}

#define DWFB_SHFL_CPLX(T)                                                                        \
    __device__ __forceinline__ T lane_c(T v, int src)                                          \
    {                                                                                          \
        return mkc(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));    \
    }
DWFB_SHFL_CPLX(float2)
DWFB_SHFL_CPLX(double2)
#undef DWFB_SHFL_CPLX

// M5 v (M5^dag v when DAG: the part of D local in the 4-D site, diagonal and
// fifth-dimension hop) for one 4-D site whose slices are spread over NL lanes at
// distance 32 / NL, part q holding v[j], s = q LT + j (PAD: NL LT > Ls).
template <bool DAG, bool PAD, int NL, typename R, int LT>
__device__ __forceinline__ void m5(const Spinor<R> (&v)[LT], Spinor<R> (&o)[LT], int q, int Ls, R dg, R mf)
{
    using T = cplx<R>;
    constexpr int D = 32 / NL;  // lanes between the parts of a site
    const int lane = threadIdx.x & 31;
    // spin component a(s) needs a(s+1), b(s) needs b(s-1)
    auto a = [](const Spinor<R>& x) { return DAG ? x.s0 : x.s1; };
    auto b = [](const Spinor<R>& x) { return DAG ? x.s1 : x.s0; };
    const T up = lane_c(a(v[0]), (lane + D) & 31);       // next lane's first (wraps to s = 0)
    T dn = lane_c(b(v[LT - 1]), (lane - D) & 31);        // previous lane's last
    T first = up;
    if (PAD)
    {
        const int ql = (Ls - 1) / LT, jl = Ls - 1 - ql * LT;
        first = lane_c(a(v[0]), lane & (D - 1));
        T last = b(v[0]);
#pragma unroll
        for (int j = 1; j < LT; ++j)
            if (j == jl)
                last = b(v[j]);
        last = lane_c(last, D * ql + (lane & (D - 1)));
        if (q == 0)
            dn = last;
    }
#pragma unroll
    for (int j = 0; j < LT; ++j)
    {
        const int s = q * LT + j;
        const bool top = PAD ? s == Ls - 1 : (j == LT - 1 && q == NL - 1);
        const T na = top ? first : (j + 1 < LT ? a(v[j + 1 < LT ? j + 1 : 0]) : up);
        const T nb = j > 0 ? b(v[j > 0 ? j - 1 : 0]) : dn;
        const R ca = top ? mf : R(-1), cb = (j == 0 && q == 0) ? mf : R(-1);
        Spinor<R> r{dg * v[j].s0, dg * v[j].s1};
        if (DAG)
        {
            r.s0 += ca * na;
            r.s1 += cb * nb;
        }
        else
        {
            r.s1 += ca * na;
            r.s0 += cb * nb;
        }
        o[j] = r;
    }
}

}  // namespace cl
}  // namespace dwfb
