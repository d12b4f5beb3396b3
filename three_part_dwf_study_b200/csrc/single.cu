// Persistent CG for one right-hand side, spread over the whole GPU.
//
// One solve of a 64x64x16 lattice is a few hundred sites per SM and iteration,
// so what it costs is latency: how long a grid-wide sum takes and how many of
// them an iteration needs. The batch kernels (solver.cu) pay, at each of their
// two barriers, a counter increment, a poll of the counter, a reload and sum of
// every chunk's partials by one warp and two list compactions; one iteration
// took 15 us at 64x64x16 although its arithmetic and L2 traffic need under 2.
// Here the barrier and the sum are one step (all_sum): every block publishes
// its partial sum in a slot of its own, tagged with the step's number, and
// every block reads all slots until their tags match. The scalars of the
// recurrence (alpha, beta, the stopping test) then live in registers, computed
// by every thread from the same bits. Measured (us an iteration, mixed / FP64):
// 64x64x16 15 / 15.9 on the batch kernels' two-barrier form, 6.6 / 8.6 here; 128x128x24
// 25.5 / - and 20.6 / 32.9. Steps to it at 64x64x16, mixed: fence after relaxed polls
// 12.9, one warp polling five slots a lane one after another 9.3, slots a 128-byte line
// apart 8.7, one slot per lane 7.9, the timer out of the first polls 6.7.
//
// Sites are dealt to threads once per solve: with at most 512 sites per SM each
// thread owns one site (ONE), whose neighbours and links it looks up once;
// larger lattices loop. Per iteration, with A = D2 D1 (D1 = D for D^dag D, D^dag
// for D D^dag):
//   phase 1: p = r + beta p_old (formed on the fly at every stencil point, the
//            centre stored into the other direction buffer), t = D1 p, |t|^2 | sum
//   phase 2: x += alpha p, r -= alpha D2 t, |r|^2                           | sum
// Reference algorithm: domain_wall/include/cg_solver.hpp:17-64; the mixed form
// is that of cg_mixed_kernel (FP32 iterations, FP64 reliable updates).
#include <algorithm>
#include <type_traits>

#include "persist.cuh"
#include "single.cuh"

namespace dwfb {
using namespace persist;

namespace {

// A site's neighbours and links, boundary signs folded into the links.
template <typename R>
struct SiteGeo
{
    int c, tp, tm, xp, xm, sup, sdn;
    R cup, cdn;
    cplx<R> ut, utm, ux, uxm;
};

template <typename R>
__device__ __forceinline__ SiteGeo<R> site_geo(const Lat& L, const cplx<R>* __restrict__ U, int i)
{
    SiteGeo<R> g;
    int s, t, x;
    site_coords(L, i, s, t, x);
    const int Nt = L.Nt, Nx = L.Nx;
    const int tp = (t + 1 == Nt) ? 0 : t + 1, tm = (t == 0) ? Nt - 1 : t - 1;
    const int xp = (x + 1 == Nx) ? 0 : x + 1, xm = (x == 0) ? Nx - 1 : x - 1;
    const int sb = s * L.V, here = t * Nx + x;
    g.c = i;
    g.tp = sb + tp * Nx + x;
    g.tm = sb + tm * Nx + x;
    g.xp = sb + t * Nx + xp;
    g.xm = sb + t * Nx + xm;
    g.sup = ((s + 1 == L.Ls) ? 0 : s + 1) * L.V + here;
    g.sdn = ((s == 0) ? L.Ls - 1 : s - 1) * L.V + here;
    g.cup = (s + 1 == L.Ls) ? R(L.mf) : R(-1);
    g.cdn = (s == 0) ? R(L.mf) : R(-1);
    g.ut = ((t == Nt - 1) ? R(L.bct) : R(1)) * U[here];
    g.utm = ((t == 0) ? R(L.bct) : R(1)) * U[tm * Nx + x];
    g.ux = ((x == Nx - 1) ? R(L.bcx) : R(1)) * U[L.V + here];
    g.uxm = ((x == 0) ? R(L.bcx) : R(1)) * U[L.V + t * Nx + xm];
    return g;
}

// D or D^dag at the site; ctr receives the input at the site itself.
template <bool DAG, typename R, typename Ld>
__device__ __forceinline__ Spinor<R> geo_op(const Ld& in, const SiteGeo<R>& g, const Lat& L, Spinor<R>& ctr)
{
    ctr = in.sp(g.c);
    cplx<R> up, lo;
    hop4<DAG, R>(in.sp(g.tp), in.sp(g.tm), in.sp(g.xp), in.sp(g.xm), g.ut, g.utm, g.ux, g.uxm, R(1),
                 R(1), R(1), R(1), up, lo);
    const R dg = R(L.diag);
    Spinor<R> o{dg * ctr.s0 - R(0.5) * up, dg * ctr.s1 - R(0.5) * lo};
    if (L.fifth)
    {
        if (!DAG)
        {
            o.s1 += g.cup * in.c(2 * long(g.sup) + 1);
            o.s0 += g.cdn * in.c(2 * long(g.sdn));
        }
        else
        {
            o.s1 += g.cdn * in.c(2 * long(g.sdn) + 1);
            o.s0 += g.cup * in.c(2 * long(g.sup));
        }
    }
    return o;
}

template <typename R, typename Ld>
__device__ __forceinline__ Spinor<R> geo_op(const Ld& in, const SiteGeo<R>& g, const Lat& L, bool dag,
                                            Spinor<R>& ctr)
{
    return dag ? geo_op<true, R>(in, g, L, ctr) : geo_op<false, R>(in, g, L, ctr);
}

__device__ __forceinline__ void slot_store(ulonglong2* p, double v, unsigned tag)
{
    const unsigned long long b = __double_as_longlong(v);
    const unsigned long long hi = (b & 0xffffffff00000000ull) | tag, lo = (b << 32) | tag;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(hi), "l"(lo) : "memory");
}

// Whether the slot carries `tag`; v receives its value then. Each half of the
// value shares an 8-byte word with the tag, so a half-written slot is seen. The
// load acquires: what the slot's block wrote before it published is visible
// after a load that returns true (a fence after relaxed polls costs another
// round trip to L2).
__device__ __forceinline__ bool slot_load(const ulonglong2* p, unsigned tag, double& v)
{
    unsigned long long hi, lo;
    asm volatile("ld.acquire.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(hi), "=l"(lo) : "l"(p) : "memory");
    if (unsigned(hi) != tag || unsigned(lo) != tag)
        return false;
    v = __longlong_as_double((hi & 0xffffffff00000000ull) | (lo >> 32));
    return true;
}

// Grid barrier and sum in one: on return every thread of every block holds the
// sum of v over the grid (the same bits everywhere: fixed tree per block, block
// sums in a fixed order), and sees what any block wrote to global memory before
// its own call. False (in every thread) once a wait ran past the limit or
// another block recorded an error. Two slot arrays alternate: a block may
// publish step n + 2 only after it has seen every block's step n + 1, which a
// block publishes after it has finished reading step n.
struct GridSum
{
    static constexpr int kPad = 8;   // slots a 128-byte line apart: polls spread over the L2 slices
    ulonglong2* slots;  // [2][gridDim.x][kPad], the first of each line used
    double* sm;         // [64] shared
    GridBar* bar;
    unsigned long long limit_ns;
    unsigned last;  // after this step the block waits for a tag that none writes (self test)
    unsigned tag;

    // The timer is read only now and then: a read takes about as long as the
    // message it waits for.
    __device__ __forceinline__ bool poll(const ulonglong2* p, unsigned want, double& u) const
    {
        for (int n = 0; n < 256; ++n)
            if (slot_load(p, want, u))
                return true;
        const unsigned long long t0 = globaltimer_ns();
        for (unsigned n = 1; !slot_load(p, want, u); ++n)
        {
            if (n % 64u != 0)
                continue;
            cuda::atomic_ref<int, cuda::thread_scope_device> err(bar->err);
            if (err.load(cuda::memory_order_relaxed) != 0)
                return false;
            if (globaltimer_ns() - t0 > limit_ns)
            {
                raise_error(bar, DWF_TIMEOUT);
                return false;
            }
        }
        return true;
    }

    __device__ __forceinline__ bool operator()(double& v)
    {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        const int G = int(gridDim.x);
        ulonglong2* const row = slots + (++tag & 1 ? G * kPad : 0);
        v = warp_sum(v);
        if (lane == 0)
            sm[w] = v;
        __syncthreads();
        if (w == 0)
        {
            v = warp_sum(lane < nw ? sm[lane] : 0.0);
            if (lane == 0)
            {
                __threadfence();
                slot_store(row + blockIdx.x * kPad, v, tag);
            }
        }
        // one slot per thread of the first warps: an acquiring load holds back
        // the loads behind it, so a lane with several slots would wait for them
        // one after another
        const int np = min(nw, (G + 31) >> 5);
        int bad = 0;
        if (w < np)
        {
            const unsigned want = tag <= last ? tag : 0u;
            double acc = 0.0, u = 0.0;
            for (int i = threadIdx.x; i < G && !bad; i += np * 32)
            {
                bad = poll(row + i * kPad, want, u) ? 0 : 1;
                acc += u;
            }
            acc = warp_sum(acc);
            if (lane == 0)
                sm[32 + w] = acc;
        }
        bad = __syncthreads_or(bad);
        v = sm[32];
        for (int k = 1; k < np; ++k)
            v += sm[32 + k];
        return !bad;
    }
};

__device__ void single_outputs(const SolveDesc& d, int iters, int status, double rr, double bb, int ru)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        d.out_iters[0] = iters;
        d.out_status[0] = status == RHS_ACTIVE ? DWF_NOT_CONVERGED : status;
        d.out_relres[0] = bb > 0.0 ? sqrt(rr / bb) : 0.0;
        d.out_ru[0] = ru;
    }
}

}  // namespace

template <bool MIXED, bool ONE>
__global__ void __launch_bounds__(kSingleThreads, 1) cg_single_kernel(SolveDesc d)
{
    using R = typename std::conditional<MIXED, float, double>::type;
    using T = cplx<R>;
    __shared__ double sm[64];
    const Lat& L = d.L;
    const bool dag1 = d.dag_first != 0;
    const int beg = int(blockIdx.x) * d.ch, end = min(beg + d.ch, L.nsite);
    GridSum gsum{reinterpret_cast<ulonglong2*>(d.part), sm, d.bar, d.timeout_ns,
                 d.mute && blockIdx.x + 1 == gridDim.x ? 2u : ~0u, 0u};
    const long uo = long(d.rhs_conf[0]) * d.usz;
    const double2* const U64 = d.U64 + uo;
    const T* const U = MIXED ? reinterpret_cast<const T*>(d.U32 + uo) : reinterpret_cast<const T*>(U64);
    T* const r = MIXED ? reinterpret_cast<T*>(d.r32) : reinterpret_cast<T*>(d.r);
    T* const pa = MIXED ? reinterpret_cast<T*>(d.p32) : reinterpret_cast<T*>(d.p);
    T* const pb = MIXED ? reinterpret_cast<T*>(d.p32b) : reinterpret_cast<T*>(d.p2);
    T* const t = MIXED ? reinterpret_cast<T*>(d.t32) : reinterpret_cast<T*>(d.t);
    T* const x = MIXED ? reinterpret_cast<T*>(d.e32) : reinterpret_cast<T*>(d.x);  // iterate or correction
    const bool on = beg + int(threadIdx.x) < end;
    SiteGeo<R> g1{};
    if (ONE && on)
        g1 = site_geo<R>(L, U, beg + int(threadIdx.x));
    // f(site) over this thread's sites
    auto sites = [&](auto f) {
        if (ONE)
        {
            if (on)
                f(beg + int(threadIdx.x));
        }
        else
            for (int i = beg + int(threadIdx.x); i < end; i += int(blockDim.x))
                f(i);
    };
    auto geo = [&](int i) { return ONE ? g1 : site_geo<R>(L, U, i); };

    // ---- r = b - A x, p = r ----
    double s0 = 0.0, s1 = 0.0;
    if (d.has_guess)
    {
        sites([&](int i) {
            st_spinor(d.t, i, op_site<double>(d, dag1, d.x, U64, i));
        });
        double z = 0.0;
        if (!gsum(z))
            return;
    }
    sites([&](int i) {
        const Spinor<double> b = ld_spinor(d.b, i);
        Spinor<double> v = b;
        if (d.has_guess)
        {
            const Spinor<double> a = op_site<double>(d, !dag1, d.t, U64, i);
            v = {b.s0 - a.s0, b.s1 - a.s1};
        }
        s0 += spinor_norm2(b);
        s1 += spinor_norm2(v);
        if constexpr (MIXED)
        {
            const Spinor<float> v32 = to32(v);
            st_spinor(r, i, v32);
            st_spinor(pa, i, v32);
            st_spinor(x, i, Spinor<float>{make_float2(0.f, 0.f), make_float2(0.f, 0.f)});
        }
        else
        {
            st_spinor(r, i, v);
            st_spinor(pa, i, v);
        }
    });
    if (!gsum(s0) || !gsum(s1))
        return;
    const double bb = s0;
    double rr = s1, rru = s1, beta = 0.0;
    int iters = 0, ru = 0, stalls = 0;
    int state = (bb == 0.0 || converged_now(d, rr, bb)) ? DWF_OK : RHS_ACTIVE;

    for (int it = 1; it <= d.maxiter && state == RHS_ACTIVE; ++it)
    {
        T* const pc = (it & 1) ? pa : pb;
        const T* const po = (it & 1) ? pb : pa;
        // phase 1
        double a0 = 0.0;
        sites([&](int i) {
            const SiteGeo<R> g = geo(i);
            Spinor<R> v, ctr;
            if (it == 1)
                v = geo_op<R>(FieldLd<R>{pc}, g, L, dag1, ctr);
            else
            {
                v = geo_op<R>(DirLd<R>{r, po, R(beta)}, g, L, dag1, ctr);
                st_spinor(pc, i, ctr);
            }
            st_spinor(t, i, v);
            a0 += spinor_norm2(v);
        });
        if (!gsum(a0))
            return;
        if (MIXED ? (a0 == 0.0 || !isfinite(a0)) : a0 == 0.0)
        {
            state = MIXED ? DWF_NOT_CONVERGED : DWF_ZERO_DENOM;  // cg_solver.hpp:45-46
            iters = it;
            break;
        }
        // phase 2
        const R al = R(rr / a0);
        a0 = 0.0;
        sites([&](int i) {
            Spinor<R> ctr;
            const Spinor<R> ap = geo_op<R>(FieldLd<R>{t}, geo(i), L, !dag1, ctr);
            st_spinor(x, i, axpy(al, ld_spinor(pc, i), ld_spinor(x, i)));
            const Spinor<R> rn = axpy(-al, ap, ld_spinor(r, i));
            st_spinor(r, i, rn);
            a0 += spinor_norm2(rn);
        });
        if (!gsum(a0))
            return;
        const double rn = a0;
        if constexpr (!MIXED)
        {
            if (converged_now(d, rn, bb))
            {
                iters = d.eigen_rule ? it - 1 : it;
                state = DWF_OK;
                rr = rn;
                break;
            }
            iters = it;
            beta = rn / rr;
            rr = rn;
        }
        else
        {
            iters = it;
            const bool want = rn < d.delta * d.delta * rru || converged_now(d, rn, bb) || it == d.maxiter;
            beta = rn / rr;
            rr = rn;
            if (!want)
                continue;
            // reliable update: t = D1 (x + e) in FP64, x + e parked in d.r;
            // then x = x + e, r = b - D2 t, e = 0
            sites([&](int i) {
                int ss, tt, xx;
                site_coords(L, i, ss, tt, xx);
                const SumLd xe{d.x, d.e32};
                const Spinor<double> v = dag1 ? dirac_site_ld<true, double>(xe, U64, L, ss, tt, xx)
                                              : dirac_site_ld<false, double>(xe, U64, L, ss, tt, xx);
                st_spinor(d.t, i, v);
                st_spinor(d.r, i, xe.sp(i));
            });
            double z = 0.0;
            if (!gsum(z))
                return;
            z = 0.0;
            sites([&](int i) {
                const Spinor<double> xn = ld_spinor(d.r, i);
                const Spinor<double> a = op_site<double>(d, !dag1, d.t, U64, i);
                const Spinor<double> b = ld_spinor(d.b, i);
                st_spinor(d.x, i, xn);
                const Spinor<double> v = {b.s0 - a.s0, b.s1 - a.s1};
                st_spinor(r, i, to32(v));
                st_spinor(x, i, Spinor<float>{make_float2(0.f, 0.f), make_float2(0.f, 0.f)});
                z += spinor_norm2(v);
            });
            if (!gsum(z))
                return;
            ru += 1;
            beta *= z / rr;  // beta = |r_new|^2 / |r_old|^2 with the replaced residual
            stalls = (z >= 0.5 * rru) ? stalls + 1 : 0;
            rr = z;
            rru = z;
            if (converged_now(d, z, bb))
                state = DWF_OK;
            else if (!isfinite(z) || stalls >= d.stall_limit || it == d.maxiter)
                state = DWF_NOT_CONVERGED;
        }
    }
    single_outputs(d, iters, state, rr, bb, ru);
}

size_t single_part_doubles(int nsm) { return size_t(4) * GridSum::kPad * size_t(nsm); }

cudaError_t load_single(bool mixed)
{
    cudaFuncAttributes a;
    const cudaError_t e = mixed ? cudaFuncGetAttributes(&a, &cg_single_kernel<true, true>)
                                : cudaFuncGetAttributes(&a, &cg_single_kernel<false, true>);
    if (e != cudaSuccess)
        return e;
    return mixed ? cudaFuncGetAttributes(&a, &cg_single_kernel<true, false>)
                 : cudaFuncGetAttributes(&a, &cg_single_kernel<false, false>);
}

cudaError_t launch_single(SolveDesc& d, bool mixed, int nsm, cudaStream_t stream, cudaEvent_t before)
{
    // one block per SM at most (the blocks wait on one another); one site per
    // thread while a block's share fits, in blocks of at least 128 threads
    const int share = (d.L.nsite + nsm - 1) / nsm;
    const bool one = share <= kSingleThreads;
    const int threads = one ? std::max(128, (share + 31) / 32 * 32) : kSingleThreads;
    d.ch = one ? threads : share;
    d.nch = (d.L.nsite + d.ch - 1) / d.ch;
    d.expected_blocks = unsigned(d.nch);
    const void* fn = mixed ? (one ? reinterpret_cast<const void*>(&cg_single_kernel<true, true>)
                                  : reinterpret_cast<const void*>(&cg_single_kernel<true, false>))
                           : (one ? reinterpret_cast<const void*>(&cg_single_kernel<false, true>)
                                  : reinterpret_cast<const void*>(&cg_single_kernel<false, false>));
    cudaError_t e = cudaMemsetAsync(d.part, 0, single_part_doubles(d.nch) * sizeof(double), stream);
    if (e == cudaSuccess && before)
        e = cudaEventRecord(before, stream);
    if (e != cudaSuccess)
        return e;
    void* args[] = {&d};
    return cudaLaunchCooperativeKernel(fn, dim3(unsigned(d.nch)), dim3(unsigned(threads)), args, 0, stream);
}

}  // namespace dwfb
