// gf_kernels.cuh -- kernel templates shared by the plugin entry points (reference layout, in
// place) and the batched engine (packed layout): parity pass, gauge quality with a deterministic
// FP64 reduction, reprojection and random start.
#pragma once

#include "gf_field.cuh"

namespace gfb {

// functional normalisation 1/(Nc*Nd), Coulomb 1/(Nc*(Nd-1)) (LandauKernelsSU3.hxx:79-82,
// CoulombKernelsSU3.hxx:75-78); theta is normalised by 1/Nc
__host__ __device__ constexpr double prefactor_gff_dev(int gauge) { return gauge == COULOMB ? 1.0 / 9.0 : 1.0 / 12.0; }

// ---- one parity pass ---------------------------------------------------------------------------
// 4 lanes per site (lane = 8*mu + site-in-warp), 8 sites per warp.  Vh is a multiple of 8 for
// even extents, so a warp is either fully inside the parity half or fully outside.
// Fup holds the up links and every down link except, for COULOMB, the temporal down link, which
// comes from the slice t-1 field Fdw at the same spatial site (CoulombKernelsSU3.hxx:226-234).
// TRACK_W (batched Coulomb): the mu = 0 planes of a timeslice hold W(x), the gauge transformation
// accumulated at that site, instead of temporal links.  Lane mu = 0 left-multiplies W by every g
// (W <- g W) and has no down link; the temporal links themselves are transformed once, at the end,
// as U_0(t,x) <- W(t,x) U_0(t,x) W(t+1,x)^dagger (the product of the reference's per-sweep left and
// right multiplications, CoulombKernelsSU3.hxx:226-247), so timeslices share no memory while they
// sweep.
// state: where given, the pass leaves the sites alone unless *state is want_state.
// W columns of the refine mode: float2 planes W[(k*3 + r)*V + s] = W(s)_{r,k}; lane mu < 3 of a
// site carries column mu through the three subgroup steps (W <- g W), lane 3 carries none.
template <typename R, int GAUGE, int ALGO, class F, bool TRACK_W = false, bool SITE_W = false>
__device__ __forceinline__ void parity_pass_warp(const F &Fup, const F &Fdw, const Geom &g, int64_t warp, int parity,
                                                 const AlgoParams &p, float2 *Wsite = nullptr,
                                                 const int *state = nullptr, int want_state = 0)
{
    const int now = state ? *state : want_state;
    const int lane = threadIdx.x & 31;
    const int mu = lane >> 3;
    const int64_t h = warp * 8 + (lane & 7);
    int32_t c[4];
    site_coords(g, h, parity, c);
    const int64_t s = h + (parity ? g.Vh : 0);
    const bool tdown = (GAUGE == COULOMB) && (mu == 0);
    const bool wlane = TRACK_W && tdown;
    const int64_t sd = tdown ? s : neighbour_down(g, c, mu);
    R ru[12], rd[12];
    Fup.load12(s, mu, ru);
    if (wlane) {  // the identity's rows; not stored
#pragma unroll
        for (int k = 0; k < 12; k++) rd[k] = (k == 0 || k == 8) ? (R)1 : (R)0;
    } else if (tdown) {
        Fdw.load12(sd, mu, rd);
    } else {
        Fup.load12(sd, mu, rd);
    }
    if (now != want_state) return;  // (an instance that is not swept in this precision; warp-uniform)
    Link<R> up, dn;
    unpack12(up, ru);
    reconstruct(up);
    unpack12(dn, rd);
    reconstruct(dn);
    Rng<R> rng;
    if (ALGO == ALG_SA || ALGO == ALG_SR || ALGO == ALG_RANDOM) rng.init(ref_rng_tid(h), p.seed, p.counter);
    Cx<R> wcol[3];
    if (SITE_W) {
        const int k = mu & 1;  // lanes mu = 0, 1 own columns 0, 1 of W; 2, 3 re-read them
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const float2 v = Wsite[(int64_t)(k * 3 + r) * g.V + s];
            wcol[r] = cx<R>((R)v.x, (R)v.y);
        }
    }
    site_update<GAUGE, ALGO, R, SITE_W>(up, dn, mu, p, rng, &wcol);
    store_link<R>(Fup, s, mu, up);
    if (SITE_W && mu < 2) {
#pragma unroll
        for (int r = 0; r < 3; r++) Wsite[(int64_t)(mu * 3 + r) * g.V + s] = make_float2((float)wcol[r].x, (float)wcol[r].y);
    }
    if (wlane) return;
    if (tdown)
        store_link<R>(Fdw, sd, mu, dn);
    else
        store_link<R>(Fup, sd, mu, dn);
}

template <typename R, int GAUGE, int ALGO, class F>
__global__ void __launch_bounds__(128) k_parity_pass(F Fup, F Fdw, Geom g, int parity, AlgoParams p)
{
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp * 8 >= g.Vh) return;
    parity_pass_warp<R, GAUGE, ALGO>(Fup, Fdw, g, warp, parity, p);
}

// One parity pass over the sites of timeslices [t_begin, t_end) only (4D gauges): in the
// parity-split order those sites are the contiguous run h in [t_begin Vs/2, t_end Vs/2), so the
// warps cover that run from its 8-aligned start and leave the sites outside it alone.  A t-slab
// rank updates its interior slices with it while the boundary links are on their way.
template <typename R, int GAUGE, int ALGO, class F>
__global__ void __launch_bounds__(128) k_parity_pass_range(F f, Geom g, int parity, AlgoParams p, int64_t h_lo,
                                                           int64_t h_hi, int64_t rng_site_offset)
{
    static_assert(GAUGE != COULOMB, "timeslice ranges are for the 4D gauges");
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, mu = lane >> 3;
    const int64_t h0 = (h_lo & ~(int64_t)7) + warp * 8;
    if (h0 >= h_hi) return;  // warp-uniform
    const int64_t h = h0 + (lane & 7);
    const bool active = h >= h_lo && h < h_hi;  // the same for the 4 lanes of a site
    int64_t s = 0, sd = 0;
    Link<R> up, dn;
    if (active) {
        int32_t c[4];
        site_coords(g, h, parity, c);
        s = h + (parity ? g.Vh : 0);
        sd = neighbour_down(g, c, mu);
        load_link<R>(f, s, mu, up);
        load_link<R>(f, sd, mu, dn);
    } else {  // no coupling: the update leaves these (unstored) links alone
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) up.e[i][j] = dn.e[i][j] = cx<R>((R)0, (R)0);
    }
    Rng<R> rng;
    if (ALGO == ALG_SA || ALGO == ALG_SR || ALGO == ALG_RANDOM)
        rng.init(ref_rng_tid(h + rng_site_offset), p.seed, p.counter);  // the whole lattice's stream for a part of it
    site_update<GAUGE, ALGO>(up, dn, mu, p, rng);
    if (active) {
        store_link<R>(f, s, mu, up);
        store_link<R>(f, sd, mu, dn);
    }
}

// Two lanes per site (site_update_pair), 16 sites per warp, over the sites h in [h_lo, h_hi) of a
// parity -- the whole of it, or the run of some timeslices: lane role of a site, 0 or 1, holds
// directions 2 role and 2 role + 1, so the SU(2) update is computed twice per site instead of four
// times.  Sites outside the range leave their lanes idle, with links that couple to nothing.  Site h
// draws the random numbers of site h + rng_site_offset.  Odd parities run from the last site to the first,
// so the second pass of a sweep begins on the links the first one left in L2.
// All four links of a lane are loaded before any arithmetic (in FP64 one link after the other, each
// followed by its third row, took 208 us per 32^4 pass with the same 8 warps per SM).  32^4, us per pass,
// against persistent passes with four lanes per site that looked one tile ahead: OR FP32 61.8 / 78.1 (0.99
// of the copy peak on 768 B per site update, part of them from L2), FP64 136 / 173 (0.90 on 1536 B); walked
// forwards in both parities 67.8 and 142.  The heat bath, whose
// rejection loop costs more than the rest of the update, Landau at T = 0.4 / U1xU1 at T = 1: FP32 128 / 226 us
// against 203 / 6078 us for a lane-wise loop with four lanes per site, FP64 272 / 380 against 387 / 7840 us.
template <typename R, int GAUGE, int ALGO, class F, int MINB>
__global__ void __launch_bounds__(128, MINB) k_parity_pass_pair(F Fup, F Fdw, Geom g, int parity, AlgoParams p,
                                                                int64_t h_lo, int64_t h_hi, int64_t rng_site_offset)
{
    const int lane = threadIdx.x & 31, role = lane >> 4;
    const int64_t h0 = h_lo & ~(int64_t)7, nwarps = (h_hi - h0 + 15) / 16;
    int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= nwarps) return;
    if (parity) warp = nwarps - 1 - warp;
    const int64_t h = h0 + warp * 16 + (lane & 15);
    const bool active = h >= h_lo && h < h_hi;
    if (!__any_sync(0xffffffffu, active)) return;
    const int64_t s = h + (parity ? g.Vh : 0);
    int64_t sd[2] = {0, 0};
    R ru[2][12] = {}, rd[2][12] = {};
    if (active) {
        int32_t c[4];
        site_coords(g, h, parity, c);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int mu = 2 * role + j;
            const bool tdown = GAUGE == COULOMB && mu == 0;  // the temporal down link is in slice t-1
            sd[j] = tdown ? s : neighbour_down(g, c, mu);
            Fup.load12(s, mu, ru[j]);
            (tdown ? Fdw : Fup).load12(sd[j], mu, rd[j]);
        }
    }
    PairLinks<R> links;
    links.set(ru, rd);
    Rng<R> rng;
    if (ALGO == ALG_SA || ALGO == ALG_SR || ALGO == ALG_RANDOM)
        rng.init(ref_rng_tid(h + rng_site_offset), p.seed, p.counter);
    links.template update<GAUGE, ALGO, false>(role, p, rng);
    if (!active) return;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int mu = 2 * role + j;
        links.rows_up(j, ru[j]);
        Fup.store12(s, mu, ru[j]);
        links.rows_dn(j, rd[j]);
        (GAUGE == COULOMB && mu == 0 ? Fdw : Fup).store12(sd[j], mu, rd[j]);
    }
}

// ---- gauge quality ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ void rows_f64(const R r[12], Link<double> &L)
{
    double d[12];
#pragma unroll
    for (int k = 0; k < 12; k++) d[k] = (double)r[k];
    unpack12(L, d);
    reconstruct(L);
}

template <typename R, class F>
__device__ __forceinline__ void load_link_f64(const F &f, int64_t s, int mu, Link<double> &L)
{
    R r[12];
    f.load12(s, mu, r);
    rows_f64(r, L);
}

// Visit the up link U_mu(x), then the down link U_mu(x - mu), of every direction mu = MU0 .. 3, in FP64
// and in that order.  The next rows are loaded before the current link's arithmetic -- the next
// direction's two links of an FP32 field, the next link of an FP64 field, 24 registers each -- and the
// loop is not unrolled, so no more than that is ever held and two blocks of 256 share an SM.  Bound by
// latency (loads and the serial FP64 chain of a link), not by DRAM.  32^4: FP32 142 -> 101 us (all eight
// links loaded at once held over 128 registers), FP64 on the reference layout 161 -> 153 us; MAG 48^4
// FP32 723 -> 472 us.
template <typename R, int MU0, class F, class Up, class Down>
__device__ __forceinline__ void visit_site_links(const F &f, const Geom &g, int64_t s, const int32_t c[4], Up up,
                                                 Down down)
{
    R ru[12], rd[12];
    f.load12(s, MU0, ru);
    if constexpr (sizeof(R) == 4) f.load12(neighbour_down(g, c, MU0), MU0, rd);
#pragma unroll 1
    for (int mu = MU0; mu < 4; mu++) {
        Link<double> l;
        if constexpr (sizeof(R) == 4) {
            const int next = mu < 3 ? mu + 1 : mu;
            R nu[12], nd[12];
            f.load12(s, next, nu);
            f.load12(neighbour_down(g, c, next), next, nd);
            rows_f64(ru, l);
            up(l);
            rows_f64(rd, l);
            down(l);
#pragma unroll
            for (int k = 0; k < 12; k++) {
                ru[k] = nu[k];
                rd[k] = nd[k];
            }
        } else {
            f.load12(neighbour_down(g, c, mu), mu, rd);
            rows_f64(ru, l);
            up(l);
            f.load12(s, mu < 3 ? mu + 1 : mu, ru);
            rows_f64(rd, l);
            down(l);
        }
    }
}

// Per-site functional and theta, computed in FP64 from the stored rows:
//  LANDAU/U1XU1 (LandauKernelsSU3.hxx:114-191, U1xU1KernelsSU3.hxx:114-191) and COULOMB
//  (CoulombKernelsSU3.hxx:110-183, mu = 1..3): gff = sum_mu Re tr U_mu(x);
//  theta = sum_ij |(A - A^dagger)_ij|^2, A = D - tr(D)/3, D = sum_mu U_mu(x) - U_mu(x-mu).
//  A - A^dagger is antihermitian, so only its three upper off-diagonal elements and the imaginary part of
//  its diagonal are summed: 9 numbers instead of D's 18, which is what lets two blocks share an SM.
//  MAG (MAGKernelsSU3.hxx:116-223): gff = sum_mu sum_j |U_mu(x)_jj|^2, theta = sum_k |X_k|.
template <int GAUGE, typename R, class F>
__device__ __forceinline__ void quality_site(const F &f, const Geom &g, int64_t s, double &gff, double &th)
{
    const int parity = s >= g.Vh;
    int32_t c[4];
    site_coords(g, s - (parity ? g.Vh : 0), parity, c);
    gff = 0;
    if (GAUGE == MAG) {
        double X[3][2] = {{0, 0}, {0, 0}, {0, 0}};
        visit_site_links<R, 0>(
            f, g, s, c,
            [&](const Link<double> &u) {
                gff += abs2(u.e[0][0]) + abs2(u.e[1][1]) + abs2(u.e[2][2]);
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;  // (0,1), (0,2), (1,2)
                    const Cx<double> a = u.e[i][i], b = u.e[i][j], cc = u.e[j][i], e = u.e[j][j];
                    // up: m00 conj(m10) - m01 conj(m11)
                    X[k][0] += (a.x * cc.x + a.y * cc.y) - (b.x * e.x + b.y * e.y);
                    X[k][1] += (a.y * cc.x - a.x * cc.y) - (b.y * e.x - b.x * e.y);
                }
            },
            [&](const Link<double> &d) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
                    // down, hermitian submatrix: conj(d_ii) d_ij - conj(d_ji) d_jj
                    const Cx<double> p = d.e[i][i], q = d.e[i][j], r = d.e[j][i], t = d.e[j][j];
                    X[k][0] += (p.x * q.x + p.y * q.y) - (r.x * t.x + r.y * t.y);
                    X[k][1] += (p.x * q.y - p.y * q.x) - (r.x * t.y - r.y * t.x);
                }
            });
        th = sqrt(X[0][0] * X[0][0] + X[0][1] * X[0][1]) + sqrt(X[1][0] * X[1][0] + X[1][1] * X[1][1]) +
             sqrt(X[2][0] * X[2][0] + X[2][1] * X[2][1]);
    } else {
        double off[3][2] = {{0, 0}, {0, 0}, {0, 0}}, diag[3] = {0, 0, 0};
        visit_site_links<R, GAUGE == COULOMB ? 1 : 0>(
            f, g, s, c,
            [&](const Link<double> &u) {
                gff += u.e[0][0].x + u.e[1][1].x + u.e[2][2].x;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
                    // (D - D^dagger)_ij = D_ij - conj(D_ji)
                    off[k][0] += u.e[i][j].x - u.e[j][i].x;
                    off[k][1] += u.e[i][j].y + u.e[j][i].y;
                    diag[k] += u.e[k][k].y;
                }
            },
            [&](const Link<double> &d) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
                    off[k][0] -= d.e[i][j].x - d.e[j][i].x;
                    off[k][1] -= d.e[i][j].y + d.e[j][i].y;
                    diag[k] -= d.e[k][k].y;
                }
            });
        const double tr = (diag[0] + diag[1] + diag[2]) / 3.0;
        double acc = 0, dd = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            acc += off[k][0] * off[k][0] + off[k][1] * off[k][1];
            const double t = diag[k] - tr;
            dd += t * t;
        }
        th = 2.0 * acc + 4.0 * dd;  // ij and ji; (2 Im)^2
    }
}

// Fixed-order block reduction (warp butterfly, then warps in order): deterministic for a fixed
// launch shape.  Result valid in thread 0.
template <int NT>
__device__ __forceinline__ void block_reduce2(double &a, double &b, bool b_is_max)
{
    __shared__ double sa[NT / 32], sb[NT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        const double ob = __shfl_xor_sync(0xffffffffu, b, o);
        b = b_is_max ? fmax(b, ob) : b + ob;
    }
    const int w = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        sa[w] = a;
        sb[w] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = sa[0];
        b = sb[0];
#pragma unroll
        for (int k = 1; k < NT / 32; k++) {
            a += sa[k];
            b = b_is_max ? fmax(b, sb[k]) : b + sb[k];
        }
    }
}

struct QualityOut {
    double *partials;    // 2 doubles per block, or null: per-site values only
    unsigned int *ticket; // zero before the launch; the last block resets it
    double *result;      // [0] = functional, [1] = theta (normalised as the reference does)
    double *gff_site;    // optional per-site arrays (generateGaugeQualityPerSite), may be null
    double *theta_site;
};

// GaugeFixingStats::generateGaugeQuality (GaugeFixingStats.hxx:186-232) in one launch: per-site
// values, per-block partial sums, and the last block to finish sums the partials in block
// order and applies the normalisation gff*preG/V, theta*preA (/V for AVERAGE).
// With o.partials null only the per-site arrays are written.
template <int GAUGE, typename R, class F, int NT = 256>
__global__ void __launch_bounds__(NT, 2) k_quality(F f, Geom g, QualityOut o, int stop_max, double preG, double preA)
{
    const int64_t s = (int64_t)blockIdx.x * NT + threadIdx.x;
    double gv = 0, tv = 0;
    if (s < g.V) {
        quality_site<GAUGE, R>(f, g, s, gv, tv);
        if (o.gff_site) o.gff_site[s] = gv;
        if (o.theta_site) o.theta_site[s] = tv;
    }
    if (!o.partials) return;
    block_reduce2<NT>(gv, tv, stop_max != 0);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        o.partials[2 * blockIdx.x] = gv;
        o.partials[2 * blockIdx.x + 1] = tv;
        __threadfence();
        last = atomicAdd(o.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double G = 0, T = 0;
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += NT) {
        G += __ldcg(&o.partials[2 * k]);
        const double t = __ldcg(&o.partials[2 * k + 1]);
        T = stop_max ? fmax(T, t) : T + t;
    }
    block_reduce2<NT>(G, T, stop_max != 0);
    if (threadIdx.x == 0) {
        double gn = G * preG / (double)g.V;
        double tn = T * preA;
        if (!stop_max) tn = tn / (double)g.V;
        o.result[0] = gn;
        o.result[1] = tn;
        *o.ticket = 0;
    }
}

// ---- reprojection (SU3::projectSU3, lattice/SU3.hxx:536-583) in FP64 ---------------------------
__device__ __forceinline__ void project_rows(Link<double> &L)
{
    double nu = 0;
#pragma unroll
    for (int i = 0; i < 3; i++) nu += abs2(L.e[0][i]);
    nu = 1.0 / sqrt(nu);
#pragma unroll
    for (int i = 0; i < 3; i++) L.e[0][i] = cx<double>(L.e[0][i].x * nu, L.e[0][i].y * nu);
    Cx<double> sp = cx<double>(0, 0);  // sum_i row1_i conj(row0_i)
#pragma unroll
    for (int i = 0; i < 3; i++) {
        sp.x += L.e[1][i].x * L.e[0][i].x + L.e[1][i].y * L.e[0][i].y;
        sp.y += L.e[1][i].y * L.e[0][i].x - L.e[1][i].x * L.e[0][i].y;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const Cx<double> t = cmul(L.e[0][i], sp);
        L.e[1][i].x -= t.x;
        L.e[1][i].y -= t.y;
    }
    double nv = 0;
#pragma unroll
    for (int i = 0; i < 3; i++) nv += abs2(L.e[1][i]);
    nv = 1.0 / sqrt(nv);
#pragma unroll
    for (int i = 0; i < 3; i++) L.e[1][i] = cx<double>(L.e[1][i].x * nv, L.e[1][i].y * nv);
    reconstruct(L);
}

template <typename R>
__global__ void __launch_bounds__(256) k_project_ref(RefField<R> f)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 4 * f.V) return;
    const int mu = (int)(idx / f.V);
    const int64_t s = idx - mu * f.V;
    Link<double> L;
    load_link_f64<R>(f, s, mu, L);
    project_rows(L);
    Link<R> o;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) o.e[i][j] = cx<R>((R)L.e[i][j].x, (R)L.e[i][j].y);
    f.store18(s, mu, o);
}

// ---- random start (COMKSU3::setHot, CommonKernelsSU3.hxx:92-130) -------------------------------
template <int I, int J, typename R>
__device__ __forceinline__ void hot_subgroup(Link<R> &M, Rng<R> &rng)
{
    R q[4];
    q[0] = (R)(rng.rand() * 2.0 - 1.0);
    q[1] = (R)(rng.rand() * 2.0 - 1.0);
    q[2] = (R)(rng.rand() * 2.0 - 1.0);
    q[3] = (R)(rng.rand() * 2.0 - 1.0);
    const R det = rsq(q[0] * q[0] + q[3] * q[3] + q[2] * q[2] + q[1] * q[1]);  // Quaternion::projectSU2
    q[0] *= det;
    q[1] *= det;
    q[2] *= det;
    q[3] *= det;
    right_mult<I, J>(M, q);
}

template <typename R>
__global__ void __launch_bounds__(256) k_set_hot_ref(RefField<R> f, uint32_t seed, uint32_t counter)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= f.V) return;
    Rng<R> rng;
    rng.init((uint32_t)s, seed, counter);
#pragma unroll 1
    for (int mu = 0; mu < 4; mu++) {
        Link<R> M;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) M.e[i][j] = cx<R>(i == j ? (R)1 : (R)0, (R)0);
        hot_subgroup<0, 1>(M, rng);
        hot_subgroup<0, 2>(M, rng);
        hot_subgroup<1, 2>(M, rng);
        f.store18(s, mu, M);
    }
}

}  // namespace gfb
