// Even-odd Schur mixed CG with one thread-block cluster per right-hand side
// and the FP32 Krylov fields resident in the cluster's registers and shared
// memory.
//
// The grid-wide kernel (cg_eo_mixed_kernel) runs every right-hand side of a
// batch in lock step: five grid barriers per iteration across all blocks, the
// FP32 fields streaming through L2. Here a cluster of CS CTAs owns one
// right-hand side at a time; CTA c holds time rows [c R, (c+1) R) (R = ceil(Nt /
// CS), the last CTA may hold fewer) of every field for every fifth-dimension
// slice. Right-hand sides are independent, so clusters never wait for one
// another; each takes the right-hand sides cluster_id, cluster_id + nclusters, ...
//
// Per iteration (FP32; the same algebra as cg_eo_mixed_kernel), each phase ended
// by a block barrier and begun by a wait for the neighbouring CTAs' rows:
//   P1 (even sites)  y = M5^-1 H_eo p
//   P2 (odd sites)   t = M5 p - H_oe y, |t|^2
//   P3 (even sites)  y = M5^dag^-1 H^dag_eo t
//   P4 (odd sites)   Ap = M5^dag t - H^dag_oe y; e += alpha p; r -= alpha Ap, |r|^2
//   P5 (odd sites)   p = r + beta p
// Shared-memory bandwidth, issue and the latency of the exchanges bound it, so
//   - only what a neighbour reads is stored in shared memory: NL = 2 or 4 threads
//     own one 4-D site of each parity, LT = ceil(Ls / NL) slices each, and keep p, r
//     and (EREG) e of the odd site in registers; M5's fifth-dimension neighbours
//     come from the thread's own registers and two shuffles. Shared memory holds
//     two fields, each with one halo row either side: A carries p (read in P1)
//     and, from P2 on, t (read in P3 and, by its owner, in P4); B carries y;
//   - lane D q + i of a warp (D = 32 / NL) holds part q of site D w + i, so every
//     quarter warp reads 128 consecutive bytes;
//   - halo rows and sums go by asynchronous remote stores counted on mbarriers
//     (cluster.cuh), so a phase waits for its own CTA (block barrier), in the edge
//     rows for the neighbouring rows, and for the sums just before their use.
// A sender may overwrite a halo row once the thread that read it has sent its own
// row of the same or a later phase back, which every phase waits for: the threads
// of the first and last row of a CTA send to, and wait for, the same neighbour.
//
// 64x64x16, 28 right-hand sides, 443 iterations each (seven clusters of 16, one B200):
// 28.4 ms with five fields in shared memory, a lane order whose 16-byte reads met
// on the same banks four ways, a cluster barrier per phase and remote gathers for
// the sums; 20.6 with p, r, e in registers; 17.6 with asynchronous stores instead of
// cluster barriers; 16.2 with sums per CTA and no timer read in the waits (a read of
// the global timer takes about a message's time); 15.1 with fewer reliable updates and
// no square roots in the stopping test; 14.4 with y and t at the thread's own places
// kept in registers between the phases (EREG: a quarter of the hops' loads). ncu (256
// threads, 60 iterations): 3.3 k instructions per warp and iteration, issue 35 % of its
// peak and shared-memory wavefronts 47 % before that last step, stalls split
// between shared-memory latency and the exchanges' waits. (These with the stop at
// twice the tolerance; at the tolerance itself it is 456 iterations and one reliable
// update more.) 64x96x16 with 56, which the grid-wide kernel had to take, 113 ms there
// and 45.5 here at equal stops.
//
// M5^-1 (per spin an Ls x Ls bidiagonal matrix with the m_f corner, closed form
// in eo.cuh): the two fifth-dimension recurrences run over the thread's slices in
// place, the threads' carries are a suffix and a prefix sum with geometric weights
// c^-k (c = 3 - M5 >= 1) over the site's threads by shuffles, and one multiply-add
// per slice adds carry and corner term. Ls that does not fill its threads (PAD)
// leaves slices at the end of the last ones zero.
//
// Reliable updates (FP64, fields x, b, t64, y64 in global memory) recompute the
// residual of the Schur normal equation from x + e when the FP32 residual has
// fallen by delta^2 since the last one, or convergence is in sight.
#include <algorithm>
#include <vector>

#include "cluster.cuh"
#include "cluster_launch.cuh"
#include "context.cuh"
#include "eo.cuh"
#include "persist.cuh"

namespace dwfb {

namespace {

namespace cg = cooperative_groups;

constexpr size_t kClHead = cl::head_bytes(cl::sum_bytes(3) + 8 * 8);  // sum tables, mbarriers, Meet

struct ClDesc
{
    int CS, R;     // CTAs per cluster, time rows per CTA
    int Nt, Nx, Nxh, Vh, Ls;
    int SS;        // float4 per slice of a shared field: (R + 2) Nxh
    float pw32[13];            // c^-k, k = 0 .. 12 (within a thread's slices)
    float q32[4];              // m_f / (1 + m_f c^-Ls) c^-(LT q): corner weight of the down form per part
    float u32[4];              // the same of the up form: ... c^-(Ls - LT q - LT)
    float pad32;               // c^(NL LT - Ls)
    double pw64[13], q64[4], u64[4], pad64;
    double delta;              // reliable-update trigger
};

__device__ __forceinline__ Spinor<float> f4s(float4 v)
{
    return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float4 s2f4(const Spinor<float>& v)
{
    return make_float4(v.s0.x, v.s0.y, v.s1.x, v.s1.y);
}

// The corner and carry weights of one lane's slices (q = the lane's part).
template <typename R>
struct M5w
{
    const R* pw;   // c^-k
    R qd, qu;      // corner weights (ClDesc q*, u* at q)
    R pad;
};

// y = M5^-1 z (M5^dag^-1 when DAG) for one 4-D site, z scaled by c^-1 already,
// its slices spread over NL lanes at distance D = 32 / NL (part q holds z[j], s = q
// LT + j, zero where s >= Ls). Up form (spin DAG ? 0 : 1): y(s)
// = U(s) - m_f y0 c^-(Ls-s), U(s) = sum_{k>=s} z(k) c^-(k-s), y0 = U(0) / (1 +
// m_f c^-Ls). Down form (the other spin): y(s) = D(s) - m_f yL c^-(s+1), D(s) =
// sum_{k<=s} z(k) c^-(s-k), yL = D(Ls-1) / (1 + m_f c^-Ls). All lanes of the warp
// take part.
template <bool DAG, bool PAD, int NL, typename R, int LT>
__device__ __forceinline__ void cl_m5inv(Spinor<R> (&z)[LT], int q, const M5w<R>& w)
{
    using T = cplx<R>;
    constexpr int D = 32 / NL;  // lanes between the parts of a site
    const R ci = w.pw[1];
#pragma unroll
    for (int j = LT - 2; j >= 0; --j)
    {
        if (DAG)
            z[j].s0 += ci * z[j + 1].s0;
        else
            z[j].s1 += ci * z[j + 1].s1;
    }
#pragma unroll
    for (int j = 1; j < LT; ++j)
    {
        if (DAG)
            z[j].s1 += ci * z[j - 1].s1;
        else
            z[j].s0 += ci * z[j - 1].s0;
    }
    const int lane = threadIdx.x & 31;
    const T zero = mkc(R(0), R(0));
    T B = DAG ? z[0].s0 : z[0].s1;            // U at the part's first slice
    T E = DAG ? z[LT - 1].s1 : z[LT - 1].s0;  // D at its last
    R cL = w.pw[LT];
#pragma unroll
    for (int step = 1; step < NL; step *= 2)
    {
        const T u = cl::lane_c(B, (lane + step * D) & 31), v = cl::lane_c(E, (lane - step * D) & 31);
        B += cL * (q + step < NL ? u : zero);  // suffix scan
        E += cL * (q >= step ? v : zero);      // prefix scan
        cL *= cL;
    }
    T cu = cl::lane_c(B, (lane + D) & 31), cd = cl::lane_c(E, (lane - D) & 31);
    const T S = cl::lane_c(B, lane & (D - 1));              // U(0)
    T Sp = cl::lane_c(E, (NL - 1) * D + (lane & (D - 1)));  // D(Ls-1), decayed by the padding
    if (PAD)
        Sp = w.pad * Sp;
    cu = (q + 1 < NL ? cu : zero) - w.qu * S;
    cd = (q > 0 ? cd : zero) - w.qd * Sp;
#pragma unroll
    for (int j = 0; j < LT; ++j)
    {
        if (DAG)
        {
            z[j].s0 += w.pw[LT - j] * cu;
            z[j].s1 += w.pw[j + 1] * cd;
        }
        else
        {
            z[j].s1 += w.pw[LT - j] * cu;
            z[j].s0 += w.pw[j + 1] * cd;
        }
    }
}

// Where the hop neighbours of a thread's 4-D site sit in a shared field of the other
// parity (slice 0; every slice is SS further), halo rows included: t +- 1, and of the
// two x neighbours the one that is not the thread's own place (t, k). The other one
// is, so the thread that owns both sites has it in registers.
struct ClNbr
{
    int tp, tm, oth;
};

// sg = +1 where the own place is the x + 1 neighbour, -1 where it is x - 1.
__device__ __forceinline__ ClNbr cl_nbr(int Nxh, int tl, int k, float sg)
{
    const int row = (tl + 1) * Nxh;
    return {row + Nxh + k, row - Nxh + k, row + (sg > 0.f ? (k == 0 ? Nxh - 1 : k - 1) : (k + 1 == Nxh ? 0 : k + 1))};
}

// The four link phases of the hops from (t, x), FP32, boundary signs folded in
// (exact: the signs are +-1): t + 1, t - 1, then the own and the other x neighbour
// with the backward one conjugated.
struct ClLinks
{
    float2 t, tm, own, oth;
};

__device__ __forceinline__ ClLinks cl_links(const float2* __restrict__ U, const Lat& L, int t, int x, float sg)
{
    const int Nt = L.Nt, Nx = L.Nx;
    const int tm = (t == 0) ? Nt - 1 : t - 1;
    const int xm = (x == 0) ? Nx - 1 : x - 1;
    const float stp = (t == Nt - 1) ? float(L.bct) : 1.f;
    const float stm = (t == 0) ? float(L.bct) : 1.f;
    const float sxp = (x == Nx - 1) ? float(L.bcx) : 1.f;
    const float sxm = (x == 0) ? float(L.bcx) : 1.f;
    const float2 fw = sxp * U[L.V + t * Nx + x], b = U[L.V + t * Nx + xm];
    const float2 bw = make_float2(sxm * b.x, -sxm * b.y);
    return {stp * U[t * Nx + x], stm * U[tm * Nx + x], sg > 0.f ? fw : bw, sg > 0.f ? bw : fw};
}

// Adds the x hop from the neighbour v on side sk (+1 forward, times k) with link u: the
// projected half-spinor and its two rows as in hop4, the side a multiplier so that
// forward and backward need no selection.
__device__ __forceinline__ void cl_xhop(const Spinor<float>& v, float2 u, float sk, float2& up, float2& lo)
{
    const float2 h = make_float2(v.s0.x + sk * v.s1.y, v.s0.y - sk * v.s1.x);
    const float2 w = cmul(u, h);
    up += w;
    lo.x -= sk * w.y;
    lo.y += sk * w.x;
}

// The hop sum of one slice (times -1/2: H) from a shared field at slice offset so; vo
// is the own place's spinor, sg its side.
template <bool DAG>
__device__ __forceinline__ Spinor<float> cl_hop(const float4* f, const ClNbr& n, const ClLinks& u, float sg, int so,
                                                const Spinor<float>& vo)
{
    constexpr float k = DAG ? 1.f : -1.f;
    const Spinor<float> a = f4s(f[n.tp + so]), b = f4s(f[n.tm + so]), c = f4s(f[n.oth + so]);
    float2 w = cmul(u.t, a.s0 + k * a.s1);
    float2 up = w, lo = k * w;
    w = cmulc(u.tm, b.s0 - k * b.s1);
    up += w;
    lo += -k * w;
    cl_xhop(vo, u.own, k * sg, up, lo);
    cl_xhop(c, u.oth, -k * sg, up, lo);
    return {up, lo};
}

// H (H^dag when DAG) times -1/2 at (s, t, x) of the other parity's global FP64 field.
template <bool DAG>
__device__ __forceinline__ Spinor<double> cl_hop64(const double2* __restrict__ f, const double2* __restrict__ U,
                                                   const Lat& L, int Nxh, long sb, int t, int x)
{
    const int Nt = L.Nt, Nx = L.Nx;
    const int tp = (t + 1 == Nt) ? 0 : t + 1, tm = (t == 0) ? Nt - 1 : t - 1;
    const int xp = (x + 1 == Nx) ? 0 : x + 1, xm = (x == 0) ? Nx - 1 : x - 1;
    double2 up, lo;
    hop4<DAG, double>(ld_spinor(f, sb + tp * Nxh + (x >> 1)), ld_spinor(f, sb + tm * Nxh + (x >> 1)),
                      ld_spinor(f, sb + t * Nxh + (xp >> 1)), ld_spinor(f, sb + t * Nxh + (xm >> 1)),
                      U[t * Nx + x], U[tm * Nx + x], U[L.V + t * Nx + x], U[L.V + t * Nx + xm],
                      (t == Nt - 1) ? L.bct : 1.0, (t == 0) ? L.bct : 1.0, (x == Nx - 1) ? L.bcx : 1.0,
                      (x == 0) ? L.bcx : 1.0, up, lo);
    return {-0.5 * up, -0.5 * lo};
}

// M5 (M5^dag when DAG) at slice s of the odd 4-D site h of a global FP64 field.
template <bool DAG>
__device__ __forceinline__ Spinor<double> cl_m5_64(const double2* __restrict__ f, const Lat& L, int Ls, long Vh,
                                                   int s, long h)
{
    const Spinor<double> c = ld_spinor(f, s * Vh + h);
    Spinor<double> o{L.diag * c.s0, L.diag * c.s1};
    const int sup = (s + 1 == Ls) ? 0 : s + 1, sdn = (s == 0) ? Ls - 1 : s - 1;
    const double cup = (s + 1 == Ls) ? L.mf : -1.0, cdn = (s == 0) ? L.mf : -1.0;
    if (!DAG)
    {
        o.s1 += cup * ld_spinor(f, sup * Vh + h).s1;
        o.s0 += cdn * ld_spinor(f, sdn * Vh + h).s0;
    }
    else
    {
        o.s1 += cdn * ld_spinor(f, sdn * Vh + h).s1;
        o.s0 += cup * ld_spinor(f, sup * Vh + h).s0;
    }
    return o;
}

// Phase timer of the cluster's first thread, kept per right-hand side in shared
// memory; the longest right-hand side's times and counts of this launch are reported
// in ph[16, 32), which eo_phase_add_kernel adds to the running totals.
struct ClClock
{
    unsigned long long* ph;  // null: off
    unsigned long long* sm;  // [15]: time of the last mark, ns and counts per phase
    __device__ __forceinline__ void start() const
    {
        if (!ph)
            return;
        for (int k = 1; k < 15; ++k)
            sm[k] = 0;
        sm[0] = globaltimer_ns();
    }
    __device__ __forceinline__ void mark(int k) const
    {
        if (!ph)
            return;
        const unsigned long long now = globaltimer_ns();
        sm[1 + k] += now - sm[0];
        sm[8 + k] += 1;
        sm[0] = now;
    }
    __device__ __forceinline__ void report() const
    {
        if (!ph)
            return;
        for (int k = 0; k < 7; ++k)
        {
            atomicMax(ph + 16 + k, sm[1 + k]);
            atomicMax(ph + 24 + k, sm[8 + k]);
        }
    }
};

// A thread's place: part q of 4-D site h of each parity in its CTA's rows.
struct ClPlace
{
    int q, h, tl, k, t, xe, xo;
    bool on;
};

template <int NL>
__device__ __forceinline__ ClPlace cl_place(const ClDesc& c, int rank)
{
    ClPlace w;
    const int t0 = rank * c.R, rows = min(c.R, c.Nt - t0);
    constexpr int D = 32 / NL;
    w.q = int(threadIdx.x & 31) / D;
    w.h = (int(threadIdx.x) >> 5) * D + int(threadIdx.x & (D - 1));
    w.on = w.h < rows * c.Nxh;
    w.tl = w.on ? w.h / c.Nxh : 0;
    w.k = w.on ? w.h - w.tl * c.Nxh : 0;
    w.t = t0 + w.tl;
    w.xe = 2 * w.k + (w.t & 1);
    w.xo = 2 * w.k + ((w.t + 1) & 1);
    return w;
}

// Reliable update in FP64 of right-hand side jr: r = b - Dhat^dag Dhat x with x
// in global memory (complete before the call); r in FP32 to d.r32 at the thread's
// own places, |r|^2 of them returned. Kept out of line: it runs once in tens of
// iterations, and its FP64 temporaries must not take the loop's registers.
template <int LT, int NL, bool PAD>
__device__ __noinline__ double cl_reliable(const EoDesc& e, const ClDesc& c, int rank, int jr, const cl::Meet meet)
{
    if (meet(false, c.CS))
        return -1.0;
    const SolveDesc& d = e.d;
    const Lat& L = d.L;
    const ClPlace w = cl_place<NL>(c, rank);
    const int Ls = c.Ls, Nxh = c.Nxh, s0 = w.q * LT;
    const long Vh = c.Vh, h64 = long(w.t) * Nxh + w.k;
    const double2* const U64 = d.U64 + long(d.rhs_conf[jr]) * d.usz;
    const double2* const xj = d.x + jr * d.fsz;
    double2* const t64 = d.t + jr * d.fsz;
    double2* const y64 = e.y64 + jr * d.fsz;
    const M5w<double> w64{c.pw64, c.q64[w.q], c.u64[w.q], c.pad64};
    const double ci = c.pw64[1];
    auto act = [&](int j) { return w.on && (!PAD || s0 + j < Ls); };
    // y64 = M5^-1 H_eo f (M5^dag^-1 H^dag_eo f)
    auto hopinv = [&](auto DAG, const double2* f) {
        constexpr bool dag = decltype(DAG)::value;
        Spinor<double> z[LT];
#pragma unroll
        for (int j = 0; j < LT; ++j)
        {
            z[j] = {mkc(0.0, 0.0), mkc(0.0, 0.0)};
            if (act(j))
            {
                const Spinor<double> v = cl_hop64<dag>(f, U64, L, Nxh, (s0 + j) * Vh, w.t, w.xe);
                z[j] = {ci * v.s0, ci * v.s1};
            }
        }
        cl_m5inv<dag, PAD, NL, double, LT>(z, w.q, w64);
#pragma unroll
        for (int j = 0; j < LT; ++j)
            if (act(j))
                st_spinor(y64, (s0 + j) * Vh + h64, z[j]);
    };
    hopinv(std::false_type{}, xj);
    cl::sync_global();
#pragma unroll 2
    for (int j = 0; j < LT; ++j)
        if (act(j))
        {
            const Spinor<double> m = cl_m5_64<false>(xj, L, Ls, Vh, s0 + j, h64);
            const Spinor<double> hy = cl_hop64<false>(y64, U64, L, Nxh, (s0 + j) * Vh, w.t, w.xo);
            st_spinor(t64, (s0 + j) * Vh + h64, Spinor<double>{m.s0 - hy.s0, m.s1 - hy.s1});
        }
    cl::sync_global();
    hopinv(std::true_type{}, t64);
    cl::sync_global();
    double a0 = 0.0;
#pragma unroll 2
    for (int j = 0; j < LT; ++j)
        if (act(j))
        {
            const Spinor<double> m = cl_m5_64<true>(t64, L, Ls, Vh, s0 + j, h64);
            const Spinor<double> hy = cl_hop64<true>(y64, U64, L, Nxh, (s0 + j) * Vh, w.t, w.xo);
            const Spinor<double> b = ld_spinor(d.b + jr * d.fsz, (s0 + j) * Vh + h64);
            const Spinor<double> v{b.s0 - (m.s0 - hy.s0), b.s1 - (m.s1 - hy.s1)};
            st_spinor(d.r32 + jr * d.fsz, (s0 + j) * Vh + h64, persist::to32(v));
            a0 += spinor_norm2(v);
        }
    return a0;
}

}  // namespace

// LT slices per thread, NL threads per site, PAD: NL LT > Ls; EREG: e in registers
// (else in shared memory). Blocks of up to MAXT threads.
template <int LT, int NL, bool PAD, bool EREG, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) cg_eo_cluster_kernel(const __grid_constant__ EoDesc e,
                                                                           const __grid_constant__ ClDesc c)
{
    const SolveDesc& d = e.d;
    const Lat& L = d.L;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const int CS = c.CS, Nxh = c.Nxh, SS = c.SS, Ls = c.Ls;
    const int cid = int(blockIdx.x) / CS, ncl = int(gridDim.x) / CS;
    const int rows = min(c.R, c.Nt - rank * c.R);
    const int prev = (rank + CS - 1) % CS, next = (rank + 1) % CS;
    const int prows = min(c.R, c.Nt - prev * c.R);
    __shared__ unsigned long long clk_sm[15];
    extern __shared__ __align__(128) unsigned char cl_smem[];
    double* const tab = reinterpret_cast<double*>(cl_smem);
    const unsigned bars = cl::smem_addr(cl_smem + cl::sum_bytes(3));  // sums, then halos [A, B][from prev, next]
    const unsigned hbar = bars + 3 * 8;
    float4* const FA = reinterpret_cast<float4*>(cl_smem + kClHead);
    float4* const ES = FA + 2 * Ls * SS;                              // !EREG: e, [LT][threads]
    float2* const LK = reinterpret_cast<float2*>(ES + (EREG ? 0 : LT * int(blockDim.x)));  // links [even, odd][4][sites]
    const cl::Sum sum{tab, tab + 3 * cl::kMaxCtas, bars, CS, rank};
    const cl::Meet meet{bars + 7 * 8};
    // lane D q + i of warp w (D = 32 / NL): part q of 4-D site D w + i of each parity
    const ClPlace pl = cl_place<NL>(c, rank);
    const int q = pl.q, tl = pl.tl, k = pl.k, t = pl.t;
    const bool on = pl.on;
    const int hs = pl.h;
    const float sge = (t & 1) ? -1.f : 1.f, sgo = -sge;  // the own place's side, even and odd site
    const ClNbr en = cl_nbr(Nxh, tl, k, sge), od = cl_nbr(Nxh, tl, k, sgo);
    const int own = (tl + 1) * Nxh + k;
    const int s0 = q * LT;
    // halo rows: a first row is the previous CTA's row after its last, a last
    // row the next CTA's row before its first
    const bool first = on && tl == 0, last = on && tl == rows - 1;
    const unsigned toprev = cl::map(cl::smem_addr(FA + (prows + 1) * Nxh + k), prev);
    const unsigned tonext = cl::map(cl::smem_addr(FA + k), next);
    const unsigned barprev = cl::map(hbar + 8, prev), barnext = cl::map(hbar, next);
    const int fB = Ls * SS;  // field B behind field A
    auto act = [&](int j) { return on && (!PAD || s0 + j < Ls); };
    // The slice stride, opaque: the compiler would otherwise hoist every slice's
    // address of every phase out of the iteration and spill them.
    auto stride = [&] {
        int x = SS;
        asm volatile("" : "+r"(x));
        return x;
    };
    // v[j] into field A (f = 0) or B (f = fB) at the thread's own place, and to the
    // CTAs that hold it as a halo row
    auto store = [&](int f, const Spinor<float> (&v)[LT]) {
        const int ss = stride();
        if (on)
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (!PAD || s0 + j < Ls)
                    FA[f + (s0 + j) * ss + own] = s2f4(v[j]);
        if (first)
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (!PAD || s0 + j < Ls)
                    cl::send(toprev + unsigned(f + (s0 + j) * ss) * 16u, s2f4(v[j]), barprev + (f ? 16u : 0u));
        if (last)
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (!PAD || s0 + j < Ls)
                    cl::send(tonext + unsigned(f + (s0 + j) * ss) * 16u, s2f4(v[j]), barnext + (f ? 16u : 0u));
    };
    // Parities of the barriers: bits 0-2 sums, 3 and 4 the halos of A and B.
    unsigned par = 0;
    int bad = 0;
    auto ran_out = [] {};
    // Wait for the halo rows this thread reads from field A (f = 0) or B.
    auto halo = [&](int f) {
        const unsigned b = hbar + 16u * f, ph = (par >> (3 + f)) & 1u;
        if (threadIdx.x == 0 && !bad)
        {
            cl::bar_expect(b, unsigned(Ls * Nxh) * 16u);
            cl::bar_expect(b + 8u, unsigned(Ls * Nxh) * 16u);
        }
        // one lane per warp polls for its warp's rows
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
        par ^= 8u << f;
    };
    auto total = [&](int slot) {
        const double v = sum.get(slot, (par >> slot) & 1u, d.timeout_ns, bad, ran_out);
        par ^= 1u << slot;
        return v;
    };
    if (threadIdx.x == 0)
    {
        for (int i = 0; i < 7; ++i)
            cl::bar_init(bars + 8u * i, i < 3 && rank + 1 == CS ? (d.mute >> i) & 1u : 0u);
        meet.init();
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cl::sync();
    // !EREG has 80 registers a thread: keep the compiler from holding the next
    // slice's neighbours while this one's are in use (24 warps hide the latency)
    auto fence = [] {
        if (!EREG)
            asm volatile("" ::: "memory");
    };
    const int nsite = int(blockDim.x) / NL;
    auto links = [&](int i) -> ClLinks {  // 0: even site, 1: odd site
        const float2* const o = LK + i * 4 * nsite + hs;
        return {o[0], o[nsite], o[2 * nsite], o[3 * nsite]};
    };
    auto eslot = [&](int j) -> float4& { return ES[j * int(blockDim.x) + int(threadIdx.x)]; };
    const M5w<float> w32{c.pw32, c.q32[q], c.u32[q], c.pad32};
    const float dg = float(L.diag), mf = float(L.mf);
    const float zs = -0.5f * c.pw32[1];  // hop factor and c^-1 of M5^-1's input
    const Spinor<float> zero{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const long fh = d.fsz, Vh = c.Vh;
    const long h64 = long(t) * Nxh + k;
    const ClClock clk{threadIdx.x == 0 && rank == 0 ? e.phase_ns : nullptr, clk_sm};

    for (int jr = cid; jr < d.nrhs; jr += ncl)
    {
        // the four links of each of the thread's sites: one copy per site, read
        // back by its lanes in each phase (16 registers otherwise)
        if (on && q < 2)
        {
            const ClLinks u = cl_links(d.U32 + long(d.rhs_conf[jr]) * d.usz, L, t, q == 0 ? pl.xe : pl.xo,
                                       q == 0 ? sge : sgo);
            float2* const o = LK + q * 4 * nsite + hs;
            o[0] = u.t;
            o[nsite] = u.tm;
            o[2 * nsite] = u.own;
            o[3 * nsite] = u.oth;
        }
        __syncwarp();
        // ---- x = 0: r = b (FP32 copy in global memory, field A p = 0); |b|^2 ----
        double a0 = 0.0;
#pragma unroll 1
        for (int j = 0; j < LT; ++j)
            if (act(j))
            {
                const Spinor<double> b = ld_spinor(d.b + jr * fh, (s0 + j) * Vh + h64);
                st_spinor(d.r32 + jr * fh, (s0 + j) * Vh + h64, persist::to32(b));
                FA[(s0 + j) * SS + own] = make_float4(0.f, 0.f, 0.f, 0.f);
                a0 += spinor_norm2(b);
            }
        sum.part(2, a0);
        __syncthreads();
        if (threadIdx.x < 32)
            sum.send(2);
        const double bb = total(2);
        double rr = bb, rru = bb, cf = 0.0;
        int it = 0, ru = 0, stalls = 0;
        int state = (bb == 0.0 || persist::converged_now(d, rr, bb) || d.maxiter < 1) ? DWF_OK : RHS_ACTIVE;
        if (state == DWF_OK && !(bb == 0.0 || persist::converged_now(d, rr, bb)))
            state = DWF_NOT_CONVERGED;

        if (__syncthreads_or(bad))
            state = cl::kGaveUp;
        clk.start();
        // Between two reliable updates: p and r come from memory (p from field
        // A's own places), e starts at zero.
        while (state == RHS_ACTIVE)
        {
            Spinor<float> p[LT], r[LT], ev[EREG ? LT : 1];
#pragma unroll
            for (int j = 0; j < LT; ++j)
            {
                p[j] = act(j) ? f4s(FA[(s0 + j) * SS + own]) : zero;
                r[j] = act(j) ? ld_spinor(d.r32 + jr * fh, (s0 + j) * Vh + h64) : zero;
                if (!EREG)
                    eslot(j) = make_float4(0.f, 0.f, 0.f, 0.f);
                else
                    ev[EREG ? j : 0] = zero;
            }
            // P5 of the iteration before
            auto direction = [&] {
                const float beta = float(cf);
#pragma unroll
                for (int j = 0; j < LT; ++j)
                    p[j] = persist::axpy(beta, p[j], r[j]);
                store(0, p);
            };
            direction();
            // One barrier ends every iteration, whether it goes on or not, and tells all
            // warps whether a wait of one of them ran out.
            bool lost = __syncthreads_or(bad) != 0, want = lost, zden = false;
            clk.mark(6);
            while (!want)
            {
                ++it;
                // (EREG) y and t at the own places, kept from the phase that forms them
                // for the phases that read them: a quarter of the hops' loads
                Spinor<float> yk[EREG ? LT : 1], tk[EREG ? LT : 1];
                // P1: y = M5^-1 H_eo p
                halo(0);
                {
                    const ClLinks u = links(0);
                    const int ss = stride();
                    Spinor<float> z[LT];
#pragma unroll
                    for (int j = 0; j < LT; ++j)
                        z[j] = zero;
                    if (on)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            if (!PAD || s0 + j < Ls)
                            {
                                const Spinor<float> v = cl_hop<false>(FA, en, u, sge, (s0 + j) * ss, p[j]);
                                z[j] = {zs * v.s0, zs * v.s1};
                                fence();
                            }
                    cl_m5inv<false, PAD, NL, float, LT>(z, q, w32);
                    store(fB, z);
                    if (EREG)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            yk[EREG ? j : 0] = z[j];
                }
                __syncthreads();
                clk.mark(0);
                // P2: t = M5 p - H_oe y, |t|^2
                halo(1);
                a0 = 0.0;
                {
                    const ClLinks u = links(1);
                    const int ss = stride();
                    Spinor<float> m[LT];
                    cl::m5<false, PAD, NL>(p, m, q, Ls, dg, mf);
                    if (on)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            if (!PAD || s0 + j < Ls)
                            {
                                const Spinor<float> v = cl_hop<false>(
                                    FA, od, u, sgo, fB + (s0 + j) * ss,
                                    EREG ? yk[EREG ? j : 0] : f4s(FA[fB + (s0 + j) * ss + own]));
                                m[j] = persist::axpy(0.5f, v, m[j]);
                                a0 += spinor_norm2(m[j]);
                                fence();
                            }
                    store(0, m);
                    if (EREG)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            tk[EREG ? j : 0] = m[j];
                }
                sum.part(1, a0);
                __syncthreads();
                if (threadIdx.x < 32)
                    sum.send(1);
                clk.mark(1);
                // P3: y = M5^dag^-1 H^dag_eo t
                halo(0);
                {
                    const ClLinks u = links(0);
                    const int ss = stride();
                    Spinor<float> z[LT];
#pragma unroll
                    for (int j = 0; j < LT; ++j)
                        z[j] = zero;
                    if (on)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            if (!PAD || s0 + j < Ls)
                            {
                                const Spinor<float> v = cl_hop<true>(
                                    FA, en, u, sge, (s0 + j) * ss,
                                    EREG ? tk[EREG ? j : 0] : f4s(FA[(s0 + j) * ss + own]));
                                z[j] = {zs * v.s0, zs * v.s1};
                                fence();
                            }
                    cl_m5inv<true, PAD, NL, float, LT>(z, q, w32);
                    store(fB, z);
                    if (EREG)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            yk[EREG ? j : 0] = z[j];
                }
                __syncthreads();
                clk.mark(3);
                const double tt = total(1);
                zden = tt == 0.0 || !isfinite(tt);  // ends the solve, e and r dropped
                const float al = float(rr / tt);
                clk.mark(2);
                // P4: Ap = M5^dag t - H^dag_oe y; e += alpha p; r -= alpha Ap; |r|^2
                halo(1);
                a0 = 0.0;
                {
                    const ClLinks u = links(1);
                    const int ss = stride();
                    Spinor<float> tv[LT], m[LT];
#pragma unroll
                    for (int j = 0; j < LT; ++j)
                        tv[j] = EREG ? tk[EREG ? j : 0] : act(j) ? f4s(FA[(s0 + j) * ss + own]) : zero;
                    cl::m5<true, PAD, NL>(tv, m, q, Ls, dg, mf);
                    if (on)
#pragma unroll
                        for (int j = 0; j < LT; ++j)
                            if (!PAD || s0 + j < Ls)
                            {
                                const Spinor<float> v = cl_hop<true>(
                                    FA, od, u, sgo, fB + (s0 + j) * ss,
                                    EREG ? yk[EREG ? j : 0] : f4s(FA[fB + (s0 + j) * ss + own]));
                                const Spinor<float> ap = persist::axpy(0.5f, v, m[j]);
                                if (!EREG)
                                    eslot(j) = s2f4(persist::axpy(al, p[j], f4s(eslot(j))));
                                else
                                    ev[EREG ? j : 0] = persist::axpy(al, p[j], ev[EREG ? j : 0]);
                                r[j] = persist::axpy(-al, ap, r[j]);
                                a0 += spinor_norm2(r[j]);
                                fence();
                            }
                }
                sum.part(0, a0);
                __syncthreads();
                if (threadIdx.x < 32)
                    sum.send(0);
                clk.mark(4);
                const double rn = total(0);
                want = zden || rn < c.delta * c.delta * rru || persist::converged_now(d, rn, bb) || it == d.maxiter;
                cf = rn / rr;
                rr = zden ? rr : rn;
                clk.mark(5);
                if (!want)
                    direction();
                lost = __syncthreads_or(bad) != 0;
                want = want || lost;
                clk.mark(6);
            }
            if (lost || zden)
                state = lost ? cl::kGaveUp : DWF_NOT_CONVERGED;
            if (state != RHS_ACTIVE)
                break;
            // ---- reliable update in FP64: x += e, r = b - Dhat^dag Dhat x ----
#pragma unroll
            for (int j = 0; j < LT; ++j)
                if (act(j))
                {
                    double2* const xj = d.x + jr * fh;
                    const long gi = (s0 + j) * Vh + h64;
                    const Spinor<double> xo = ld_spinor(xj, gi);
                    const Spinor<double> de = persist::to64(!EREG ? f4s(eslot(j)) : ev[EREG ? j : 0]);
                    st_spinor(xj, gi, Spinor<double>{xo.s0 + de.s0, xo.s1 + de.s1});
                    FA[(s0 + j) * SS + own] = s2f4(p[j]);
                }
            a0 = cl_reliable<LT, NL, PAD>(e, c, rank, jr, meet);
            bad |= a0 < 0.0;
            sum.part(2, a0);
            __syncthreads();
            if (threadIdx.x < 32 && !bad)
                sum.send(2);
            const double rt = total(2);
            if (__syncthreads_or(bad))
            {
                state = cl::kGaveUp;
                break;
            }
            ru += 1;
            cf = cf * (rt / rr);
            stalls = (rt >= 0.5 * rru) ? stalls + 1 : 0;
            rr = rt;
            rru = rt;
            if (persist::converged_now(d, rt, bb))
                state = DWF_OK;
            else if (!isfinite(rt) || stalls >= d.stall_limit || it == d.maxiter)
                state = DWF_NOT_CONVERGED;
            clk.mark(5);
        }
        const bool gave = state == cl::kGaveUp;
        if (gave && threadIdx.x == 0)
            raise_error(d.bar, DWF_TIMEOUT);
        clk.report();
        if (!gave && rank == 0 && threadIdx.x == 0)
        {
            d.out_iters[jr] = it;
            d.out_status[jr] = state;
            d.out_relres[jr] = bb > 0.0 ? sqrt(rr / bb) : 0.0;
            d.out_ru[jr] = ru;
        }
        // the next right-hand side overwrites the fields and partials
        if (meet.left() || meet(gave, CS))
        {
            cl::settle();
            return;
        }
    }
}

namespace {

// Kernel forms. Two threads per site hold more slices each (fewer instructions
// for places, links, sums and waits per slice, more registers a thread); four
// where Ls needs it. X(form, LT, NL, PAD, EREG, MAXT)
#define DWFB_CL_PADS(X, lt, nl, er, mt) X(lt, nl, false, er, mt) X(lt, nl, true, er, mt)
#define DWFB_CL_FORM2(X, er, mt)                                                                  \
    DWFB_CL_PADS(X, 1, 2, er, mt) DWFB_CL_PADS(X, 2, 2, er, mt) DWFB_CL_PADS(X, 3, 2, er, mt)     \
    DWFB_CL_PADS(X, 4, 2, er, mt) DWFB_CL_PADS(X, 5, 2, er, mt) DWFB_CL_PADS(X, 6, 2, er, mt)     \
    DWFB_CL_PADS(X, 7, 2, er, mt) DWFB_CL_PADS(X, 8, 2, er, mt)
// Four threads per site only where two cannot (cl_shape takes the first form that
// fits): Ls > 16, and of the smaller Ls the two below, whose links and e take a little
// less shared memory in CTAs of one or two long rows.
#define DWFB_CL_KERNELS(X)                                                                      \
    DWFB_CL_FORM2(X, true, 256) DWFB_CL_FORM2(X, false, 384)                                    \
    DWFB_CL_PADS(X, 5, 4, true, 512) DWFB_CL_PADS(X, 6, 4, true, 512)                           \
    X(3, 4, false, false, 768) X(4, 4, true, false, 768)                                        \
    DWFB_CL_PADS(X, 5, 4, false, 768) DWFB_CL_PADS(X, 6, 4, false, 768)

struct ClShape : ClusterLaunch
{
    int maxt = 0;
    bool ereg = false;
};

size_t cl_smem_bytes(const Lat& L, const ClShape& s)
{
    return kClHead + size_t(2) * L.Ls * (s.R + 2) * (L.Nx / 2) * sizeof(float4) +
           size_t(8) * (s.threads / s.NL) * sizeof(float2) +
           (s.ereg ? 0 : size_t(s.LT) * s.threads * sizeof(float4));
}

constexpr size_t kClSmemMax = 227 * 1024 - 128;  // 128 bytes are static

const void* cl_kernel(const ClShape& s, bool pad)
{
#define DWFB_CL_PICK(lt, nl, p, er, mt)                                            \
    if (s.LT == lt && s.NL == nl && pad == p && s.ereg == er && s.maxt == mt)      \
        return reinterpret_cast<const void*>(&cg_eo_cluster_kernel<lt, nl, p, er, mt>);
    DWFB_CL_KERNELS(DWFB_CL_PICK)
#undef DWFB_CL_PICK
    return nullptr;
}

// Cluster shape for a batch: the rows per CTA for which the estimated time of an
// iteration over the whole batch is least. An iteration of one cluster takes
// about 3.5 us of latencies (five phases, two sums) plus 0.09 us per warp and
// slice of a CTA at four threads per site, 0.08 at two, more where CTAs share an SM; the batch takes
// as many rounds as its right-hand sides need of the resident clusters, whose
// number falls with the CTAs per cluster (a cluster sits in one GPC: 7 clusters of
// 16 fit, 16 of 8). Measured: 64x64x16 with 28 right-hand sides 16.2 ms at 16 CTAs,
// 26 at 11; 64x32x16 with 112: 30.6 at 8 CTAs, 50 at 16; 48x40x12 with 20: 6.3 at 16
// CTAs, 6.1 at 8, 3.9 at 6; 64x96x16 with 56: two threads per site 46.4, four 54.7.
ClShape cl_shape(const dwf_ctx* c, int nrhs)
{
    const Lat& L = c->L;
    ClShape best;
    const int Nxh = L.Nx / 2;
    if (L.Ls > 24 || L.Nt % 2 != 0 || L.Nx % 2 != 0)
        return best;
    double least = 0.0;
    for (int R = L.Nt; R >= 1; --R)
    {
        const int CS = (L.Nt + R - 1) / R;
        if (CS > cl::kMaxCtas)
            break;
        if (R > 1 && (L.Nt + R - 2) / (R - 1) == CS)
            continue;  // fewer rows per CTA with as many CTAs
        for (int form = 0; form < 4; ++form)
        {
            ClShape sh;
            sh.R = R;
            sh.CS = CS;
            sh.NL = form < 2 ? 2 : 4;
            sh.LT = (L.Ls + sh.NL - 1) / sh.NL;
            sh.ereg = form % 2 == 0;
            sh.maxt = form == 0 ? 256 : form == 1 ? 384 : form == 2 ? 512 : 768;
            const int D = 32 / sh.NL;
            sh.threads = (R * Nxh + D - 1) / D * 32;
            sh.smem = cl_smem_bytes(L, sh);
            if (sh.threads > sh.maxt || sh.smem > kClSmemMax)
                continue;
            sh.fn = cl_kernel(sh, sh.NL * sh.LT != L.Ls);
            if (!sh.fn || (sh.resident = resident_clusters(sh, c->device, kClSmemMax)) < 1)
                continue;
            const int used = std::min(sh.resident, nrhs);
            const double share = std::max(1.0, double(used) * sh.CS / c->nsm);
            const double rounds = (nrhs + used - 1) / used;
            const double t = rounds * (3.5 + (sh.NL == 4 ? 0.09 : 0.08) * (sh.threads / 32) * sh.LT * share);
            if (best.CS == 0 || t < least)
            {
                best = sh;
                least = t;
            }
            break;
        }
    }
    return best;
}

}  // namespace

// Launch the cluster solver for a batch prepared by propagators_eo (fields in
// EoDesc as for cg_eo_mixed_kernel). Returns DWF_BAD_ARG (nothing launched)
// when the lattice or the device does not allow it: the caller then runs the
// grid-wide kernel. dry: only check that the cluster kernel takes this batch and
// prepare its launch; *launched tells whether it would launch, *wave (when not
// null) how many right-hand sides the resident clusters solve at once.
int launch_eo_cluster(dwf_ctx* c, EoDesc& e, bool* launched, bool dry, int* wave)
{
    *launched = false;
    const Lat& L = c->L;
    const ClShape sh = cl_shape(c, std::max(1, c->eo_shape_rhs > 0 ? c->eo_shape_rhs : e.d.nrhs));
    if (!sh.fn)
        return DWF_BAD_ARG;
    if (dry)
    {
        *launched = true;
        if (wave)
            *wave = sh.resident;
        return DWF_OK;
    }
    ClDesc cd{};
    cd.CS = sh.CS;
    cd.R = sh.R;
    cd.Nt = L.Nt;
    cd.Nx = L.Nx;
    cd.Nxh = L.Nx / 2;
    cd.Vh = L.V / 2;
    cd.Ls = L.Ls;
    cd.SS = (sh.R + 2) * cd.Nxh;
    const double cc = L.diag;
    auto pw = [&](int k) {
        double p = 1.0;
        for (int i = 0; i < std::abs(k); ++i)
            p = k > 0 ? p / cc : p * cc;
        return p;
    };
    for (int k = 0; k <= 12; ++k)
        cd.pw32[k] = float(cd.pw64[k] = pw(k));
    const double corner = L.mf / (1.0 + L.mf * pw(L.Ls));
    for (int q = 0; q < sh.NL; ++q)
    {
        cd.q32[q] = float(cd.q64[q] = corner * pw(sh.LT * q));
        cd.u32[q] = float(cd.u64[q] = corner * pw(L.Ls - sh.LT * q - sh.LT));
    }
    cd.pad32 = float(cd.pad64 = pw(L.Ls - sh.NL * sh.LT));
    // Fewer reliable updates than the grid kernel's delta of 0.1 asks for: one costs
    // about four iterations here. 64x64x16, 28 right-hand sides to 1e-12: 0.1 -> 12
    // updates, 16.2 ms; 0.03 -> 8, 15.5; 0.01 -> 6, 15.2; 24x20x8 needs 184, 188, 190
    // iterations there, and 213 at 0.003. The solutions are no further off for it:
    // on eight sets from 46x18x13 to 62x94x16, mf 0.02 to 0.1, the mean errors at 1e-8,
    // 1e-10 and 1e-12 agree to 2 % with those of 0.1, at 32x32x24 to 11 %; on smaller
    // lattices, where a solve ends a few iterations apart, either is the better one (by
    // 1.4 at 24x20x8, 2.9 at most at 16x16x4).
    cd.delta = 0.02;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    sh.config(std::min(sh.resident, e.d.nrhs), c->stream, cfg, attr);
    void* args[] = {&e, &cd};
    if (cudaLaunchKernelExC(&cfg, sh.fn, args) != cudaSuccess)
        return ctx_fail(c, DWF_CUDA_ERROR, "even-odd cluster solver: launch failed");
    *launched = true;
    return DWF_OK;
}

}  // namespace dwfb
