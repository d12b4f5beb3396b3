// Full-lattice CG on D^dag D or D D^dag with one thread-block cluster per
// right-hand side, for lattices whose search direction and operator temporary
// fit a cluster's shared memory: Wilson lattices and the smaller domain-wall ones.
//
// There the grid-wide kernels are bound by the latency of their grid barriers (4.9 us
// an iteration for one right-hand side at 32x32, 16 for a batch of 16 at 48x40), however
// little there is to compute. Here CTA c of a cluster holds time rows [c R, (c+1) R)
// for every slice; NL threads own a 4-D site, LT = ceil(Ls / NL) slices each, with
// r and the iterate (FP64) or the correction e (mixed) in registers; shared memory
// holds p and t = D1 p, each with one halo row either side, exchanged by
// asynchronous stores counted on mbarriers as in eo_cluster.cu (cluster.cuh). An
// iteration is three phases, ended by block barriers only:
//   p = r + beta p | t = D1 p, |t|^2 | x += alpha p, r -= alpha D2 t, |r|^2
// (D1 = D for D^dag D, D^dag for D D^dag). A CTA's next message into a neighbour's
// halo row needs the neighbour's own row of the phase between, which its threads
// send after they have read the halo row.
//
// FP64: the reference algorithm (domain_wall/include/cg_solver.hpp:17-64; Eigen's
// stopping rule and count for Wilson). Mixed: FP32 iterations with FP64 reliable
// updates as in cg_mixed_kernel, x, b and the FP64 temporaries in global memory.
#include <algorithm>
#include <type_traits>

#include "cg_cluster.cuh"
#include "cluster.cuh"
#include "cluster_launch.cuh"
#include "persist.cuh"

namespace dwfb {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 512;
constexpr int kSlots = 4;  // sums: |r|^2, |t|^2, |b|^2 and the replaced |r|^2
constexpr size_t kHead = cl::head_bytes(cl::sum_bytes(kSlots) + (kSlots + 6) * 8);

struct CgGeo
{
    int CS, R;  // CTAs per cluster, time rows per CTA
    int SS;     // sites per slice of a shared field: (R + 2) Nx
};

// A spinor field in shared memory: FP32 one float4 per site, FP64 the two spins
// as separate planes, so that consecutive sites are consecutive 16-byte words.
template <typename R>
struct SField;
template <>
struct SField<float>
{
    float4* f;
    __device__ __forceinline__ Spinor<float> ld(int i) const
    {
        const float4 v = f[i];
        return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
    }
    __device__ __forceinline__ void st(int i, const Spinor<float>& v) const
    {
        f[i] = make_float4(v.s0.x, v.s0.y, v.s1.x, v.s1.y);
    }
};
template <>
struct SField<double>
{
    double2* f;
    int plane;
    __device__ __forceinline__ Spinor<double> ld(int i) const { return {f[i], f[plane + i]}; }
    __device__ __forceinline__ void st(int i, const Spinor<double>& v) const
    {
        f[i] = v.s0;
        f[plane + i] = v.s1;
    }
};

__device__ __forceinline__ void send_spinor(unsigned a, int, const Spinor<float>& v, unsigned bar)
{
    cl::send(a, make_float4(v.s0.x, v.s0.y, v.s1.x, v.s1.y), bar);
}
__device__ __forceinline__ void send_spinor(unsigned a, int plane, const Spinor<double>& v, unsigned bar)
{
    cl::send(a, v.s0, bar);
    cl::send(a + unsigned(plane) * 16u, v.s1, bar);
}

// A thread's place: part q of the 4-D site (t, x), row tl of its CTA.
struct CgPlace
{
    int q, h, tl, t, x;
    bool on;
};

template <int NL>
__device__ __forceinline__ CgPlace cg_place(const Lat& L, const CgGeo& g, int rank)
{
    constexpr int D = 32 / NL;
    CgPlace w;
    const int t0 = rank * g.R, rows = min(g.R, L.Nt - t0);
    w.q = int(threadIdx.x & 31) / D;
    w.h = (int(threadIdx.x) >> 5) * D + int(threadIdx.x & (D - 1));
    w.on = w.h < rows * L.Nx;
    w.tl = w.on ? w.h / L.Nx : 0;
    w.x = w.on ? w.h - w.tl * L.Nx : 0;
    w.t = t0 + w.tl;
    return w;
}

// r = b - D2 D1 x in FP64 over this thread's sites, x in global memory and complete
// before the call (d.t is scratch), the residual to d.r32 (MIXED) or d.r; returns
// the thread's share of |r|^2.
template <int LT, int NL, bool MIXED>
__device__ __noinline__ double cg_residual(const SolveDesc& d, const CgGeo& g, int rank, int jr)
{
    const Lat& L = d.L;
    const CgPlace w = cg_place<NL>(L, g, rank);
    const bool dag1 = d.dag_first != 0;
    const long f0 = long(jr) * d.fsz;
    const double2* const U = d.U64 + long(d.rhs_conf[jr]) * d.usz;
#pragma unroll 2
    for (int j = 0; j < LT; ++j)
    {
        const int s = w.q * LT + j;
        if (w.on && s < L.Ls)
            st_spinor(d.t + f0, s * L.V + w.t * L.Nx + w.x,
                      dag1 ? dirac_site<true, double>(d.x + f0, U, L, s, w.t, w.x)
                           : dirac_site<false, double>(d.x + f0, U, L, s, w.t, w.x));
    }
    cl::sync_global();
    double a = 0.0;
#pragma unroll 2
    for (int j = 0; j < LT; ++j)
    {
        const int s = w.q * LT + j;
        if (w.on && s < L.Ls)
        {
            const long i = long(s) * L.V + w.t * L.Nx + w.x;
            const Spinor<double> v = dag1 ? dirac_site<false, double>(d.t + f0, U, L, s, w.t, w.x)
                                          : dirac_site<true, double>(d.t + f0, U, L, s, w.t, w.x);
            const Spinor<double> b = ld_spinor(d.b + f0, i);
            const Spinor<double> r{b.s0 - v.s0, b.s1 - v.s1};
            if (MIXED)
                st_spinor(d.r32 + f0, i, persist::to32(r));
            else
                st_spinor(d.r + f0, i, r);
            a += spinor_norm2(r);
        }
    }
    return a;
}

}  // namespace

// MIXED: FP32 with reliable updates, else FP64. LT slices per thread, NL threads per
// site; FIFTH: the operator has the fifth-dimension hop (domain wall).
template <bool MIXED, int LT, int NL, bool FIFTH>
__global__ void __launch_bounds__(kThreads, 1) cg_cluster_kernel(const __grid_constant__ SolveDesc d,
                                                               const __grid_constant__ CgGeo g)
{
    using R = typename std::conditional<MIXED, float, double>::type;
    const Lat& L = d.L;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const int CS = g.CS, SS = g.SS, Ls = L.Ls, Nx = L.Nx, V = L.V;
    const int cid = int(blockIdx.x) / CS, ncl = int(gridDim.x) / CS;
    const int rows = min(g.R, L.Nt - rank * g.R);
    const int prev = (rank + CS - 1) % CS, next = (rank + 1) % CS;
    const int prows = min(g.R, L.Nt - prev * g.R);
    extern __shared__ __align__(128) unsigned char cg_smem[];
    double* const tab = reinterpret_cast<double*>(cg_smem);
    const unsigned bars = cl::smem_addr(cg_smem + cl::sum_bytes(kSlots));  // sums, then halos [p, t][prev, next]
    const unsigned hbar = bars + kSlots * 8;
    using W = typename std::conditional<MIXED, float4, double2>::type;
    constexpr int WPS = MIXED ? 1 : 2;  // 16-byte words per spinor
    W* const base = reinterpret_cast<W*>(cg_smem + kHead);
    const int fT = WPS * Ls * SS;  // field t behind field p
    const int plane = Ls * SS;
    auto field = [&](int f) {
        if constexpr (MIXED)
            return SField<float>{base + f};
        else
            return SField<double>{base + f, plane};
    };
    cplx<R>* const LK = reinterpret_cast<cplx<R>*>(base + 2 * fT);  // links [4][sites]
    const int nsite = int(blockDim.x) / NL;
    const cl::Sum sum{tab, tab + kSlots * cl::kMaxCtas, bars, CS, rank};
    const cl::Meet meet{bars + (kSlots + 4) * 8};
    const cl::Quit quit{meet.word + 8u};

    const CgPlace pl = cg_place<NL>(L, g, rank);
    const int q = pl.q, s0 = q * LT, tl = pl.tl, x = pl.x;
    const bool on = pl.on;
    const bool first = on && tl == 0, last = on && tl == rows - 1;
    const int own = (tl + 1) * Nx + x;
    const int nxp = (tl + 1) * Nx + (x + 1 == Nx ? 0 : x + 1), nxm = (tl + 1) * Nx + (x == 0 ? Nx - 1 : x - 1);
    const unsigned toprev = cl::map(cl::smem_addr(base + (prows + 1) * Nx + x), prev);
    const unsigned tonext = cl::map(cl::smem_addr(base + x), next);
    const unsigned barprev = cl::map(hbar + 8, prev), barnext = cl::map(hbar, next);
    const R dg = R(L.diag), mf = R(L.mf);
    const Spinor<R> zero{mkc(R(0), R(0)), mkc(R(0), R(0))};
    const long h = long(pl.t) * Nx + x;
    auto act = [&](int j) { return on && s0 + j < Ls; };
    // the slice stride, opaque so that the slices' addresses are not hoisted out of
    // the iteration and spilled
    auto stride = [&] {
        int v = SS;
        asm volatile("" : "+r"(v));
        return v;
    };
    unsigned par = 0;  // barrier parities: bits 0-3 sums, 4 and 5 the halos of p and t
    int bad = 0, it = 0;
    auto store = [&](int f, const Spinor<R> (&v)[LT]) {
        const int ss = stride();
        const SField<R> F = field(f ? fT : 0);
        if (on)
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (s0 + j < Ls)
                    F.st((s0 + j) * ss + own, v[j]);
        if (first)
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (s0 + j < Ls)
                    send_spinor(toprev + unsigned((f ? fT : 0) + (s0 + j) * ss) * 16u, plane, v[j], barprev + 16u * f);
        if (last)
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (s0 + j < Ls)
                    send_spinor(tonext + unsigned((f ? fT : 0) + (s0 + j) * ss) * 16u, plane, v[j], barnext + 16u * f);
    };
    auto ran_out = [&] { quit.from(it + 1); };
    auto halo = [&](int f) {
        const unsigned b = hbar + 16u * f, ph = (par >> (kSlots + f)) & 1u;
        if (threadIdx.x == 0 && !bad)
        {
            cl::bar_expect(b, unsigned(Ls * Nx) * unsigned(2 * sizeof(cplx<R>)));
            cl::bar_expect(b + 8u, unsigned(Ls * Nx) * unsigned(2 * sizeof(cplx<R>)));
        }
        const bool lo = __any_sync(0xffffffffu, first) || threadIdx.x == 0;
        const bool hi = __any_sync(0xffffffffu, last) || threadIdx.x == 0;
        if ((threadIdx.x & 31) == 0)
        {
            if (lo)
                cl::wait(b, ph, d.timeout_ns, bad, ran_out);
            if (hi)
                cl::wait(b + 8u, ph, d.timeout_ns, bad, ran_out);
        }
        __syncwarp();
        par ^= (1u << kSlots) << f;
    };
    auto total = [&](int slot) {
        const double v = sum.get(slot, (par >> slot) & 1u, d.timeout_ns, bad, ran_out);
        par ^= 1u << slot;
        return v;
    };
    // part(slot) of every warp, a block barrier, the CTA's sum on its way
    auto put = [&](int slot, double v) {
        sum.part(slot, v);
        __syncthreads();
        if (threadIdx.x < 32)
            sum.send(slot);
    };
    // D (D^dag when dag) of shared field f at this thread's slices
    auto apply = [&](int f, bool dag, Spinor<R> (&o)[LT]) {
        const int ss = stride();
        const SField<R> F = field(f ? fT : 0);
        cplx<R> u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            u[k] = LK[k * nsite + pl.h];
        Spinor<R> v[LT];
#pragma unroll
        for (int j = 0; j < LT; ++j)
            v[j] = act(j) ? F.ld((s0 + j) * ss + own) : zero;
        auto hop = [&](auto DAG) {
            constexpr bool dg_ = decltype(DAG)::value;
            if constexpr (FIFTH)
                cl::m5<dg_, true, NL>(v, o, q, Ls, dg, mf);
            else
            {
#pragma unroll
                for (int j = 0; j < LT; ++j)
                    o[j] = {dg * v[j].s0, dg * v[j].s1};
            }
            if (on)
#pragma unroll
                for (int j = 0; j < LT; ++j)
                    if (s0 + j < Ls)
                    {
                        const int so = (s0 + j) * ss;
                        cplx<R> up, lo;
                        hop4<dg_, R>(F.ld(so + own + Nx), F.ld(so + own - Nx), F.ld(so + nxp), F.ld(so + nxm), u[0],
                                     u[1], u[2], u[3], R(1), R(1), R(1), R(1), up, lo);
                        o[j].s0 += R(-0.5) * up;
                        o[j].s1 += R(-0.5) * lo;
                    }
        };
        if (dag)
            hop(std::true_type{});
        else
            hop(std::false_type{});
    };
    const bool dag1 = d.dag_first != 0;
    if (threadIdx.x == 0)
    {
        for (int i = 0; i < kSlots + 4; ++i)
            cl::bar_init(bars + 8u * i, i < kSlots && rank + 1 == CS ? (d.mute >> i) & 1u : 0u);
        meet.init();
        quit.init();
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cl::sync();

    for (int jr = cid; jr < d.nrhs; jr += ncl)
    {
        const long f0 = long(jr) * d.fsz;
        if (d.active_in && !d.active_in[jr])
        {
            if (rank == 0 && threadIdx.x == 0)
            {
                d.out_iters[jr] = 0;
                d.out_status[jr] = DWF_OK;
                d.out_relres[jr] = 0.0;
                d.out_ru[jr] = 0;
            }
            continue;
        }
        const auto* const U = [&] {
            if constexpr (MIXED)
                return d.U32 + long(d.rhs_conf[jr]) * d.usz;
            else
                return d.U64 + long(d.rhs_conf[jr]) * d.usz;
        }();
        if (on && q == 0)
        {
            const int t = pl.t, tm = (t == 0) ? L.Nt - 1 : t - 1, xm = (x == 0) ? Nx - 1 : x - 1;
            LK[pl.h] = ((t == L.Nt - 1) ? R(L.bct) : R(1)) * U[t * Nx + x];
            LK[nsite + pl.h] = ((t == 0) ? R(L.bct) : R(1)) * U[tm * Nx + x];
            LK[2 * nsite + pl.h] = ((x == Nx - 1) ? R(L.bcx) : R(1)) * U[V + t * Nx + x];
            LK[3 * nsite + pl.h] = ((x == 0) ? R(L.bcx) : R(1)) * U[V + t * Nx + xm];
        }
        __syncwarp();
        // ---- r = b - A x to global memory, p = 0; |b|^2, |r|^2 ----
        double a0 = 0.0, a1 = 0.0;
#pragma unroll 1
        for (int j = 0; j < LT; ++j)
            if (act(j))
            {
                const Spinor<double> b = ld_spinor(d.b + f0, long(s0 + j) * V + h);
                a0 += spinor_norm2(b);
                field(0).st((s0 + j) * SS + own, zero);
                if (!d.has_guess)
                {
                    if constexpr (MIXED)
                        st_spinor(d.r32 + f0, long(s0 + j) * V + h, persist::to32(b));
                    else
                        st_spinor(d.r + f0, long(s0 + j) * V + h, b);
                }
            }
        a1 = d.has_guess ? cg_residual<LT, NL, MIXED>(d, g, rank, jr) : a0;
        put(2, a0);
        const double bb = total(2);
        put(3, a1);
        double rr = total(3);
        double rru = rr, cf = 0.0;
        it = 0;
        int iters = 0, ru = 0, stalls = 0;
        int state = (bb == 0.0 || persist::converged_now(d, rr, bb)) ? DWF_OK : RHS_ACTIVE;

        // Mixed: one pass between two reliable updates. FP64: one pass. `gave` is the
        // same in all threads of the CTA, and so is every value taken from a sum once
        // it is false.
        bool gave = __syncthreads_or(bad) != 0;
        while (state == RHS_ACTIVE && it < d.maxiter && !gave)
        {
            Spinor<R> r[LT], xe[LT];
#pragma unroll
            for (int j = 0; j < LT; ++j)
            {
                r[j] = zero;
                xe[j] = zero;
                if (act(j))
                {
                    const long i = long(s0 + j) * V + h;
                    if constexpr (MIXED)
                        r[j] = ld_spinor(d.r32 + f0, i);
                    else
                    {
                        r[j] = ld_spinor(d.r + f0, i);
                        xe[j] = ld_spinor(d.x + f0, i);
                    }
                }
            }
            bool want = false, zden = false;
            do
            {
                ++it;
                // p = r + beta p
                {
                    const int ss = stride();
                    const R beta = R(cf);
                    Spinor<R> p[LT];
#pragma unroll
                    for (int j = 0; j < LT; ++j)
                        p[j] = act(j) ? persist::axpy(beta, field(0).ld((s0 + j) * ss + own), r[j]) : zero;
                    store(0, p);
                }
                __syncthreads();
                gave = quit.at(it);
                // t = D1 p, |t|^2
                halo(0);
                {
                    Spinor<R> o[LT];
                    apply(0, dag1, o);
                    store(1, o);
                    a0 = 0.0;
#pragma unroll
                    for (int j = 0; j < LT; ++j)
                        if (act(j))
                            a0 += spinor_norm2(o[j]);
                }
                if (gave)
                    break;
                put(1, a0);
                // x += alpha p; r -= alpha D2 t; |r|^2
                halo(1);
                Spinor<R> ap[LT];
                apply(1, !dag1, ap);
                const double tt = total(1);
                // a zero denominator ends the solve with x as it is (FP64: t = D1 p = 0
                // has a finite p, so 0 p adds nothing; mixed: e is dropped)
                zden = MIXED ? (tt == 0.0 || !isfinite(tt)) : tt == 0.0;
                const R al = zden ? R(0) : R(rr / tt);
                a0 = 0.0;
                {
                    const int ss = stride();
#pragma unroll
                    for (int j = 0; j < LT; ++j)
                        if (act(j))
                        {
                            xe[j] = persist::axpy(al, field(0).ld((s0 + j) * ss + own), xe[j]);
                            r[j] = persist::axpy(-al, ap[j], r[j]);
                            a0 += spinor_norm2(r[j]);
                        }
                }
                put(0, a0);
                const double rn = total(0);
                iters = it;
                if constexpr (MIXED)
                    want = zden || rn < d.delta * d.delta * rru || persist::converged_now(d, rn, bb) || it == d.maxiter;
                else
                {
                    if (!zden && persist::converged_now(d, rn, bb))
                    {
                        iters = d.eigen_rule ? it - 1 : it;
                        state = DWF_OK;
                    }
                    want = zden || state == DWF_OK || it == d.maxiter;
                }
                cf = rn / rr;
                rr = zden ? rr : rn;
            } while (!want);
            // (a warp whose sum ran out may be at the next iteration's first barrier)
            if (!gave)
            {
                __syncthreads();
                gave = quit.at(it + 1);
            }
            if (gave)
                break;
            if (zden)
                state = MIXED ? DWF_NOT_CONVERGED : DWF_ZERO_DENOM;  // cg_solver.hpp:45-46
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (act(j))
                {
                    const long i = long(s0 + j) * V + h;
                    if constexpr (MIXED)
                    {
                        const Spinor<double> xo = ld_spinor(d.x + f0, i), e = persist::to64(xe[j]);
                        if (state == RHS_ACTIVE)
                            st_spinor(d.x + f0, i, Spinor<double>{xo.s0 + e.s0, xo.s1 + e.s1});
                    }
                    else
                        st_spinor(d.x + f0, i, xe[j]);
                }
            if (MIXED && state == RHS_ACTIVE)
            {
                // reliable update in FP64: x += e, r = b - A x
                if (meet(false, CS))
                {
                    cl::settle();
                    return;
                }
                put(3, cg_residual<LT, NL, MIXED>(d, g, rank, jr));
                const double rt = total(3);
                gave = __syncthreads_or(bad) != 0;
                ru += 1;
                cf = cf * (rt / rr);
                stalls = (rt >= 0.5 * rru) ? stalls + 1 : 0;
                rr = rt;
                rru = rt;
                if (persist::converged_now(d, rt, bb))
                    state = DWF_OK;
                else if (!isfinite(rt) || stalls >= d.stall_limit || it == d.maxiter)
                    state = DWF_NOT_CONVERGED;
            }
        }
        if (gave && threadIdx.x == 0)
            raise_error(d.bar, DWF_TIMEOUT);
        if (!gave && rank == 0 && threadIdx.x == 0)
        {
            d.out_iters[jr] = iters;
            d.out_status[jr] = state == RHS_ACTIVE ? DWF_NOT_CONVERGED : state;
            d.out_relres[jr] = bb > 0.0 ? sqrt(rr / bb) : 0.0;
            d.out_ru[jr] = ru;
        }
        // the next right-hand side overwrites the fields and links
        if (meet(gave, CS))
        {
            cl::settle();
            return;
        }
    }
    // no CTA leaves while another may still store into its shared memory
    cl::sync();
}

namespace {

constexpr size_t kSmemMax = 227 * 1024;

// Slices per thread up to which r, the iterate and the temporaries stay in 128 registers.
constexpr int kMaxLt32 = 6, kMaxLt64 = 3;

const void* kernel_of(bool mixed, bool fifth, int LT, int NL)
{
#define DWFB_CGC(m, lt, nl, f)                             \
    if (mixed == m && fifth == f && LT == lt && NL == nl) \
        return reinterpret_cast<const void*>(&cg_cluster_kernel<m, lt, nl, f>);
#define DWFB_CGC_NL(m, lt) DWFB_CGC(m, lt, 1, true) DWFB_CGC(m, lt, 2, true) DWFB_CGC(m, lt, 4, true) DWFB_CGC(m, lt, 8, true)
    DWFB_CGC(true, 1, 1, false)
    DWFB_CGC(false, 1, 1, false)
    DWFB_CGC_NL(true, 1) DWFB_CGC_NL(true, 2) DWFB_CGC_NL(true, 3) DWFB_CGC_NL(true, 4) DWFB_CGC_NL(true, 5)
    DWFB_CGC_NL(true, 6)
    DWFB_CGC_NL(false, 1) DWFB_CGC_NL(false, 2) DWFB_CGC_NL(false, 3)
#undef DWFB_CGC_NL
#undef DWFB_CGC
    return nullptr;
}

// Estimated time (us) of an iteration over the whole batch on the grid-wide kernels
// (measured: one right-hand side 64x64x16 6.6 mixed, 8.6 FP64, 24x20x10 5.9; 28 at
// 64x64x16 89 mixed, 143 FP64, 16 at 48x40 16).
double grid_time(const Lat& L, bool mixed, int nrhs)
{
    const double sites = double(L.nsite) * nrhs;
    if (nrhs == 1)
        return 5.6 + sites * (mixed ? 1.8e-5 : 4.6e-5);
    return 14.0 + sites * (mixed ? 0.7e-4 : 1.1e-4);
}

}  // namespace

cudaError_t load_cg_cluster64()
{
    for (int LT = 1; LT <= kMaxLt64; ++LT)
        for (int NL = 1; NL <= 8; NL *= 2)
        {
            cudaFuncAttributes a;
            const cudaError_t e = cudaFuncGetAttributes(&a, kernel_of(false, true, LT, NL));
            if (e != cudaSuccess)
                return e;
        }
    return cudaSuccess;
}

// The cluster shape with the least estimated time of an iteration over the whole
// batch, if that beats the grid-wide kernels. An iteration takes about 1.4 us of
// message and sum latencies (1.8 with the fifth dimension's shuffles), plus per
// slice of a thread 0.9 us in FP64, 0.75 in FP32 (its chain of loads and products,
// twice) and 0.055 / 0.04 us per warp, so small LT and few warps win, and the batch
// takes the rounds its right-hand sides need of the resident clusters. Measured (us
// an iteration, FP64): Wilson 32x32 2.6 at 2 to 7 CTAs' rows each, 3.1 with two CTAs;
// 12x10x6 3.3 / 3.9 / 4.7 at LT 1 / 2 / 3; 24x20x10 4.6 at LT 2, 5.2 at 3; 48x40 with 16
// right-hand sides 2.8 (grid-wide 16); 40x40x8 5.0 (grid-wide 6.2).
cudaError_t launch_cg_cluster(SolveDesc& d, bool mixed, int device, int nsm, cudaStream_t stream,
                              cudaEvent_t before, bool* taken)
{
    *taken = false;
    const Lat& L = d.L;
    const bool fifth = L.fifth != 0;
    const int words = mixed ? 1 : 2;
    ClusterLaunch best;
    double least = grid_time(L, mixed, d.nrhs);
    for (int R = L.Nt; R >= 1; --R)
    {
        const int CS = (L.Nt + R - 1) / R;
        if (CS > cl::kMaxCtas)
            break;
        if (R > 1 && (L.Nt + R - 2) / (R - 1) == CS)
            continue;  // fewer rows per CTA with as many CTAs
        for (int NL = 1; NL <= 8; NL *= 2)
        {
            ClusterLaunch s;
            s.R = R;
            s.CS = CS;
            s.NL = NL;
            s.LT = (L.Ls + NL - 1) / NL;
            if (s.LT > (mixed ? kMaxLt32 : kMaxLt64) || (NL > 1 && NL >= 2 * L.Ls) || (!fifth && NL > 1))
                continue;
            const int D = 32 / NL;
            const long warps = (long(R) * L.Nx + D - 1) / D;
            if (warps * 32 > kThreads)
                continue;
            s.threads = int(warps) * 32;
            s.smem = kHead + size_t(2) * words * L.Ls * (R + 2) * L.Nx * 16 +
                     size_t(4) * (s.threads / NL) * (mixed ? sizeof(float2) : sizeof(double2));
            if (s.smem > kSmemMax)
                continue;
            s.fn = kernel_of(mixed, fifth, s.LT, NL);
            if (!s.fn || (s.resident = resident_clusters(s, device, kSmemMax)) < 1)
                continue;
            const int used = std::min(s.resident, d.nrhs);
            const double share = std::max(1.0, double(used) * CS / nsm);
            const double rounds = (d.nrhs + used - 1) / used;
            const double t = rounds * ((fifth ? 1.8 : 1.4) + s.LT * ((mixed ? 0.75 : 0.9) +
                                                                     (mixed ? 0.04 : 0.055) * double(warps) * share));
            if (t < least)
            {
                best = s;
                least = t;
            }
        }
    }
    if (best.CS == 0)
        return cudaSuccess;
    CgGeo g{best.CS, best.R, (best.R + 2) * L.Nx};
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    best.config(std::min(best.resident, d.nrhs), stream, cfg, attr);
    void* args[] = {&d, &g};
    cudaError_t e = before ? cudaEventRecord(before, stream) : cudaSuccess;
    if (e != cudaSuccess)
        return e;
    e = cudaLaunchKernelExC(&cfg, best.fn, args);
    *taken = e == cudaSuccess;
    return e;
}

}  // namespace dwfb
