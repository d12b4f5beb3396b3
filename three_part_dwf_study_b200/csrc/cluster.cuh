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

__device__ __forceinline__ void bar_init(unsigned bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
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
// CTA. One lane per warp polls: all threads polling, and a message per warp
// instead of per CTA, made the mbarrier the bottleneck (2.5 us a sum at 16 CTAs of
// 16 warps against 0.5). Thread 0 arms the slot's barrier in get(). A slot
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
    __device__ __forceinline__ bool get(int slot, unsigned parity, unsigned long long limit_ns, double& v) const
    {
        const int lane = threadIdx.x & 31;
        bool ok = true;
        if (lane == 0)
        {
            if (threadIdx.x == 0)
                bar_expect(bar + 8u * slot, unsigned(CS) * 8u);
            ok = bar_wait(bar + 8u * slot, parity, limit_ns);
        }
        __syncwarp();
        v = warp_sum(lane < CS ? tab[slot * kMaxCtas + lane] : 0.0);
        return ok;
    }
};
__host__ __device__ constexpr size_t sum_bytes(int nslot)
{
    return size_t(nslot) * (kMaxCtas + kMaxWarps) * sizeof(double);
}

// A CTA that gave up a wait stays until the others of its cluster have given up
// theirs too (each waits for it within a phase or two), so that none of them
// stores into the shared memory of a CTA that has left.
__device__ __forceinline__ void linger(unsigned long long limit_ns)
{
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 3 * limit_ns)
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
