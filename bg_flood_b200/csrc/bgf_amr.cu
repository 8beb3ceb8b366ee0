// Multi-level flow step and the bed preparation (see bgf_amr.cuh for the design).
//
// One stage (predictor or corrector) of a step on a mesh with several refinement
// levels is this chain of launches over all active blocks:
//
//   amr_halo_kernel     halo of h, u, v from the neighbours' interiors (fillHalo),
//                       wet/dry restriction next to finer blocks, zs = zb + h, and
//                       the interior gradients of h, u, v of blocks that have a
//                       finer neighbour (what the neighbour's prolongation reads)
//   amr_refine_kernel   halos next to coarser blocks rebuilt by linear
//                       reconstruction in the coarse cell (refine_linear)
//   amr_wetdry_kernel   wet/dry prolongation decisions, one launch per level
//                       above the coarsest (the reference visits blocks in order,
//                       so a decision may see a coarser block's halo that the
//                       same pass already changed)
//   amr_apply_kernel    the decisions applied (depth and bed of the parent), zs
//                       recomputed on the prolongated halo
//   amr_step_kernel     two launches (blocks without, then with finer neighbours): tile with
//                       its outer stencil ring, gradients, wet-slope reset, faces with the
//                       coarse/fine source substitution, cell dtmax and the block minimum
//                       (predictor only); faces next to finer blocks replaced by the mean of
//                       the two fine faces, boundary segments, flux divergence, advance
//                       (predictor: the tendencies; corrector: full step, friction, rain,
//                       next state, time slot)
//
// refine, wetdry and apply run on the blocks that have a coarser side only.
//
// The reference counterpart is FlowGPU/FlowCPU with its fillHalo, gradient,
// refine_linear, WetDryProlongation and HaloFlux calls (src/FlowCPU.cu:15-253).
#include <cuda_runtime.h>

#include "bgf_amr.cuh"
#include "bgf_internal.h"

#ifndef BGF_VARIANT
#define BGF_VARIANT exact
#endif

namespace bgf {
namespace BGF_VARIANT {

#include "bgf_stage.cuh"
#include "bgf_pair.cuh"
#include "bgf_quad.cuh"

__device__ __forceinline__ bool has_finer_neighbour(const int* nbr, int nbm, const int* lv, int ib)
{
    const int l = lv[ib];
    bool f = false;
#pragma unroll
    for (int k = 0; k < 8; k++) f |= lv[nbr[k * nbm + ib]] > l;
    return f;
}

// wetdryrestriction (src/ConserveElevation.cu:676-726): a halo cell next to a finer
// neighbour whose four cells are partly wet takes the depth-weighted surface of the
// wet ones minus its own bed.  h and z are those cells' depths and beds, hv the restricted
// depth from the halo fill.
template <class T> __device__ __forceinline__ T wetdry_mean(const T (&h)[4], const T (&z)[4], T eps, T zbw, T hv)
{
    const T iiwet = h[0] > eps ? (T)1.0 : (T)0.0;
    const T irwet = h[1] > eps ? (T)1.0 : (T)0.0;
    const T itwet = h[2] > eps ? (T)1.0 : (T)0.0;
    const T itrwet = h[3] > eps ? (T)1.0 : (T)0.0;
    const T cwet = (iiwet + irwet + itwet + itrwet);
    T hwet = (iiwet * h[0] + irwet * h[1] + itwet * h[2] + itrwet * h[3]);
    T zswet = (iiwet * h[0]) * (z[0] + h[0]) + (irwet * h[1]) * (z[1] + h[1]) + (itwet * h[2]) * (z[2] + h[2]) +
              (itrwet * h[3]) * (z[3] + h[3]);
    if (cwet > (T)0.0 && cwet < (T)4.0) {
        zswet = zswet / hwet;
        return ((T)0.0 < zswet - zbw) ? zswet - zbw : (T)0.0;
    }
    return hv;
}
template <class T, class HA>
__device__ __forceinline__ T wetdry_restrict(const HA& h, const Acc324<T>& zb, T eps, T zbw, int nb, int s, int j,
                                             T hv)
{
    const int jj = j < BW / 2 ? 2 * j : (j - BW / 2) * 2;
    int x0, y0;
    if (s == 0) { x0 = BW - 2; y0 = jj; }
    else if (s == 1) { x0 = 0; y0 = jj; }
    else if (s == 2) { x0 = jj; y0 = BW - 2; }
    else { x0 = jj; y0 = 0; }
    const T h4[4] = {h(nb, x0, y0), h(nb, x0 + 1, y0), h(nb, x0, y0 + 1), h(nb, x0 + 1, y0 + 1)};
    const T z4[4] = {zb(nb, x0, y0), zb(nb, x0 + 1, y0), zb(nb, x0, y0 + 1), zb(nb, x0 + 1, y0 + 1)};
    return wetdry_mean<T>(h4, z4, eps, zbw, hv);
}

// ---------------------------------------------------------------- stage state

// State of any cell as a stage reads it: state n in the predictor; in the corrector
// the half-step state h* = Advance(state n, predictor tendencies, dt / 2), rebuilt
// from the stored tendencies (the predictor advance is pointwise, so this is the
// value the reference's half-step state holds at that cell).  Blocks on one level
// among same-level neighbours run the single-level kernels, which store the same
// tendencies, so every block reads its neighbours the same way.
template <class T> struct StageState {
    const DevModel<T>& m;
    const StepParams<T>& p;
    int cur;
    bool half;
    T halfdt;
    double time;
    __device__ __forceinline__ void get(int b, int x, int y, T& ho, T& uo, T& vo) const
    {
        const size_t g = (size_t)b * 256 + y * 16 + x;
        const T hv = m.h[cur][g], uv = m.u[cur][g], vv = m.v[cur][g];
        if (!half) {
            ho = hv; uo = uv; vo = vv;
            return;
        }
        // the predictor's river source of the cell (AddRiverForcing after updateEV)
        const T dhs = add_rivers<T>(m, p, b, x, y, m.dh[g], time);
        advance<T>(halfdt, p.eps, p.eps_d, p.forcemass != 0, hv, uv, vv, dhs, m.dhu[g], m.dhv[g], ho, uo, vo);
    }
};
template <class T> struct StageComp {
    const StageState<T>& s;
    int f;
    __device__ __forceinline__ T operator()(int b, int x, int y) const
    {
        T a0, a1, a2;
        s.get(b, x, y, a0, a1, a2);
        return f == 0 ? a0 : f == 1 ? a1 : a2;
    }
};

// What a stage reads of a cell, and the state it makes of it (StageState::get in two halves,
// so that the loads of several cells are in flight while the step's dt is worked out).
template <class T> struct RawCell {
    T h, u, v, dh, dhu, dhv;
};
template <class T> __device__ __forceinline__ RawCell<T> raw_cell(const DevModel<T>& m, int cur, bool half, int b, int c)
{
    const size_t g = (size_t)b * 256 + c;
    RawCell<T> r{m.h[cur][g], m.u[cur][g], m.v[cur][g], (T)0, (T)0, (T)0};
    if (half) {
        r.dh = m.dh[g];
        r.dhu = m.dhu[g];
        r.dhv = m.dhv[g];
    }
    return r;
}
template <class T>
__device__ __forceinline__ void stage_cell(const StageState<T>& S, const RawCell<T>& r, int b, int c, T& ho, T& uo, T& vo)
{
    if (!S.half) {
        ho = r.h; uo = r.u; vo = r.v;
        return;
    }
    const T dhs = add_rivers<T>(S.m, S.p, b, c & 15, c >> 4, r.dh, S.time);
    advance<T>(S.halfdt, S.p.eps, S.p.eps_d, S.p.forcemass != 0, r.h, r.u, r.v, dhs, r.dhu, r.dhv, ho, uo, vo);
}

// ---------------------------------------------------------------- stage kernels

// 128 threads a block: 0..63 fill a halo cell each, 64..127 copy four interior cells each.
// The kernel waits on chains of dependent loads (tables, time slot, cells), so what counts is
// the blocks in flight: eight per SM.  With 320 threads (three blocks per SM) it took 108 us
// per launch on 9,834 blocks of a rain run with levels 0-2.
constexpr int HALO_THREADS = 128;

template <class T>
__global__ void __launch_bounds__(HALO_THREADS, sizeof(T) == 4 ? 8 : 5)
    amr_halo_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ AmrDev<T> a,
                    const __grid_constant__ StepParams<T> p0, int parity, int stage)
{
    __shared__ T th[3][324];
    __shared__ T s_halfdt;
    const int tid = threadIdx.x;
    const int ib = m.active[blockIdx.x];
    const int sc = scen_of(m, ib);
    const StepParams<T>& p = m.sparams ? m.sparams[sc] : p0;
    const int nbm = m.nblkmem, lev = m.level[ib];
    // the rule of the halo cell follows from the tables alone
    const int s = (tid >> 4) & 3, j = tid & 15;
    CellRule<T> r{};
    int nbh = ib, lnb = lev;
    if (tid < 64) {
        r = halo_rule<T>(m.nbr, nbm, m.level, ib, s, j);
        nbh = m.nbr[(2 * s + (j >= BW / 2 ? 1 : 0)) * nbm + ib];
        lnb = m.level[nbh];
    }
    const bool finer = has_finer_neighbour(m.nbr, nbm, m.level, ib);
    pdl_wait();
    const TimeState ts = m.time[2 * sc + parity];
    if (!step_live(ts)) return;
    const int cur = ts.cur;
    const bool half = stage != 0;
    const int nc = tid >= 64 ? 4 : r.kind == 0 ? 1 : r.kind == 2 ? 3 : 4;
    RawCell<T> q[4];
    int qb[4], qc[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        qb[k] = tid >= 64 ? ib : r.b[k];
        qc[k] = tid >= 64 ? tid - 64 + 64 * k : r.y[k] * 16 + r.x[k];
        if (k < nc) q[k] = raw_cell<T>(m, cur, half, qb[k], qc[k]);
    }
    if (half) {
        if (tid == 64) s_halfdt = step_dt<T>(ts, m.dtmin[2 * sc + parity]) * (T)0.5;
        __syncthreads();
    }
    const StageState<T> S{m, p, cur, half, half ? s_halfdt : (T)0, ts.totaltime};
    T* const* W = a.W[stage];
    const size_t base = (size_t)ib * 324;
    T c[4][3];
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (k < nc) stage_cell<T>(S, q[k], qb[k], qc[k], c[k][0], c[k][1], c[k][2]);
    if (tid >= 64) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int i = hi18(qc[k] & 15, qc[k] >> 4);
            th[0][i] = c[k][0];
            th[1][i] = c[k][1];
            th[2][i] = c[k][2];
            W[0][base + i] = c[k][0];
            W[2][base + i] = c[k][1];
            W[3][base + i] = c[k][2];
            W[1][base + i] = a.zb[base + i] + c[k][0];
        }
    } else {
        // rule_eval of the three components
        T out[3];
#pragma unroll
        for (int f = 0; f < 3; f++) {
            if (r.kind == 0) out[f] = c[0][f];
            else if (r.kind == 1) out[f] = (T)0.25 * (c[0][f] + c[1][f] + c[2][f] + c[3][f]);
            else out[f] = r.w1 * c[0][f] + r.w2 * c[1][f] + r.w3 * c[2][f];
        }
        int hx, hy;
        halo_xy(s, j, hx, hy);
        const int hc = hi18(hx, hy);
        const T zbw = a.zb[base + hc];
        if (a.wetdryfix && lnb > lev) {
            if (r.kind == 1) {
                // the four cells of the restriction are the rule's own
                T z[4], h4[4];
#pragma unroll
                for (int k = 0; k < 4; k++) z[k] = a.zb[(size_t)qb[k] * 324 + hi18(qc[k] & 15, qc[k] >> 4)];
                // (x0, y0), (x0 + 1, y0), (x0, y0 + 1), (x0 + 1, y0 + 1) among the rule's cells
                const int o = s == 0 ? 0x2301 : s == 1 ? 0x3210 : s == 2 ? 0x2031 : 0x3120;
                T zz[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int e = (o >> (4 * k)) & 3;
                    h4[k] = e == 0 ? c[0][0] : e == 1 ? c[1][0] : e == 2 ? c[2][0] : c[3][0];
                    zz[k] = e == 0 ? z[0] : e == 1 ? z[1] : e == 2 ? z[2] : z[3];
                }
                out[0] = wetdry_mean<T>(h4, zz, p.eps, zbw, out[0]);
            } else {
                out[0] = wetdry_restrict<T>(StageComp<T>{S, 0}, Acc324<T>{a.zb}, p.eps, zbw, nbh, s, j, out[0]);
            }
        }
        th[0][hc] = out[0];
        th[1][hc] = out[1];
        th[2][hc] = out[2];
        W[0][base + hc] = out[0];
        W[2][base + hc] = out[1];
        W[3][base + hc] = out[2];
        W[1][base + hc] = zbw + out[0];
    }
    // gradientC (src/Gradients.cu:921-957) of h, u, v for the prolongation of the
    // finer neighbours' halos
    pdl_trigger();
    if (!finer) return;
    __syncthreads();
    const T delta = calcres<T>(p.delta0, lev);
    const T rdelta = (T)1.0 / delta;
    for (int k = tid; k < 256; k += HALO_THREADS) {
        const int i = hi18(k & 15, k >> 4);
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const T* t = th[f];
            a.G0[2 * f][base + i] = div_by(minmod2(p.theta, t[i - 1], t[i], t[i + 1]), delta, rdelta);
            a.G0[2 * f + 1][base + i] = div_by(minmod2(p.theta, t[i - 18], t[i], t[i + 18]), delta, rdelta);
        }
    }
}

// The small kernels take four blocks of a list per CTA, 64 threads (halo cells) each; the
// parent cell follows from the tables alone and is looked up before the wait for the kernel
// before (pdl_wait).
constexpr int SIDE_BLOCKS = 4;

template <class T>
__global__ void __launch_bounds__(64 * SIDE_BLOCKS)
    amr_refine_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ AmrDev<T> a,
                      const __grid_constant__ StepParams<T> p0, const int* list, int n, int parity, int stage)
{
    const int w = blockIdx.x * SIDE_BLOCKS + (threadIdx.x >> 6);
    const int s = (threadIdx.x >> 4) & 3, j = threadIdx.x & 15;
    int ib = 0, pb, px, py;
    const bool on = w < n && parent_cell(m.nbr, m.nblkmem, m.level, ib = list[w], s, j, pb, px, py);
    pdl_wait();
    pdl_trigger();
    if (!on) return;
    const int sc = scen_of(m, ib);
    const TimeState ts = m.time[2 * sc + parity];
    if (!step_live(ts)) return;
    const StepParams<T>& p = m.sparams ? m.sparams[sc] : p0;
    int hx, hy;
    halo_xy(s, j, hx, hy);
    const size_t o = (size_t)ib * 324 + hi18(hx, hy);
    T* const* W = a.W[stage];
#pragma unroll
    for (int f = 0; f < 3; f++) {
        const int wf = f == 0 ? 0 : f + 1;  // h, u, v in W order h, zs, u, v
        W[wf][o] = refine_value<T>(Acc324<T>{W[wf]}, Acc324<T>{a.G0[2 * f]}, Acc324<T>{a.G0[2 * f + 1]}, s, j, pb, px,
                                   py, m.level[ib], p.delta0, p.delta0_d);
    }
}

// WetDryProlongation (src/ConserveElevation.cu:80-203) for the blocks of one level:
// a halo cell next to a coarser block whose parent or any of the parent's four
// neighbours is dry takes the parent's depth and bed.  The reference visits the
// blocks in active-list order and changes halos as it goes, so the four neighbours
// of a parent that lie in the coarse block's own halo are read as already changed
// when that coarse block comes earlier in the list and its decision (made by the
// launch for its level, which runs first) says so.
template <class T>
__global__ void __launch_bounds__(64 * SIDE_BLOCKS)
    amr_wetdry_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ AmrDev<T> a,
                      const __grid_constant__ StepParams<T> p0, const int* list, int n, int parity, int stage)
{
    const int w = blockIdx.x * SIDE_BLOCKS + (threadIdx.x >> 6);
    const int nbm = m.nblkmem;
    const int s = (threadIdx.x >> 4) & 3, j = threadIdx.x & 15;
    int ib = 0, pb, px, py;
    const bool on = w < n && parent_cell(m.nbr, nbm, m.level, ib = list[w], s, j, pb, px, py);
    pdl_wait();
    pdl_trigger();
    if (!on) return;
    const TimeState ts = m.time[2 * scen_of(m, ib) + parity];
    if (!step_live(ts)) return;
    const T* H = a.W[stage][0];
    const T eps = (m.sparams ? m.sparams[scen_of(m, ib)] : p0).eps;
    const bool earlier = a.rank[pb] < a.rank[ib];
    auto hval = [&](int x, int y) -> T {
        const T v = H[(size_t)pb * 324 + hi18(x, y)];
        if (!earlier) return v;
        int hs, hj;
        if (x < 0) { hs = 0; hj = y; }
        else if (x >= BW) { hs = 1; hj = y; }
        else if (y < 0) { hs = 2; hj = x; }
        else if (y >= BW) { hs = 3; hj = x; }
        else return v;
        int qb, qx, qy;
        if (!parent_cell(m.nbr, nbm, m.level, pb, hs, hj, qb, qx, qy)) return v;
        if (!a.pflag[(size_t)pb * 64 + hs * 16 + hj]) return v;
        return H[(size_t)qb * 324 + hi18(qx, qy)];
    };
    const bool dry = !(hval(px, py) > eps && hval(px - 1, py) > eps && hval(px + 1, py) > eps &&
                       hval(px, py + 1) > eps && hval(px, py - 1) > eps);
    a.pflag[(size_t)ib * 64 + s * 16 + j] = dry ? 1 : 0;
}

// The prolongation decisions applied, then RecalculateZs (src/Halo.cu:72-107) on
// the halo cells next to coarser blocks.
template <class T>
__global__ void __launch_bounds__(64 * SIDE_BLOCKS)
    amr_apply_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ AmrDev<T> a, const int* list, int n,
                     int parity, int stage)
{
    const int w = blockIdx.x * SIDE_BLOCKS + (threadIdx.x >> 6);
    const int s = (threadIdx.x >> 4) & 3, j = threadIdx.x & 15;
    int ib = 0, pb, px, py;
    const bool on = w < n && parent_cell(m.nbr, m.nblkmem, m.level, ib = list[w], s, j, pb, px, py);
    pdl_wait();
    pdl_trigger();
    if (!on) return;
    const TimeState ts = m.time[2 * scen_of(m, ib) + parity];
    if (!step_live(ts)) return;
    int hx, hy;
    halo_xy(s, j, hx, hy);
    const size_t o = (size_t)ib * 324 + hi18(hx, hy);
    const size_t po = (size_t)pb * 324 + hi18(px, py);
    T* H = a.W[stage][0];
    if (a.wetdryfix && a.pflag[(size_t)ib * 64 + s * 16 + j]) {
        H[o] = H[po];
        a.zb[o] = a.zb[po];
    }
    a.W[stage][1][o] = a.zb[o] + H[o];
}

// Resident CTAs per SM of the step kernel (launch bounds).
template <class T> struct AmrOcc {
    static constexpr int step = sizeof(T) == 4 ? 6 : 3;
};

// Cells of a pair that a thread of the step kernel owns: one in FP64, a pair in FP32 on every
// mesh (quad_lanes in bgf_flow.cu also takes one cell on small meshes of the exact build).
template <class T> __host__ __device__ constexpr int amr_lanes() { return sizeof(T) == 8 ? 1 : 2; }

// Fluxes and update of a chain's blocks, in the layout of the single-level kernels
// (bgf_quad.cuh).  The tile comes from the stage tile W (interior and ring 1, whose
// halos the chain filled) and the outer ring rules (ring 2); gradients, wet-slope reset and
// faces are the single-level kernels' own, with the coarse/fine source substitution on the
// sides whose neighbour is coarser.  Those sides' faces are all that goes to memory (a.F):
// the coarser neighbour takes their means.  pass 0 runs on the blocks without finer
// neighbours, which it finishes, and on those with finer and coarser ones, for their faces;
// pass 1 on the blocks with finer neighbours.  (One kernel wrote every face, 8.7 KB a block,
// and a second read them back with the tile: 185 us per stage on the 9,834 blocks of a
// rain run with levels 0-2.)  The same operations in the same order as the reference's
// FlowCPU: the exact build matches the oracle bit for bit.
template <class T, int ENGINE>
__global__ void __launch_bounds__(Quad<T, amr_lanes<T>()>::NT, AmrOcc<T>::step)
    amr_step_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ AmrDev<T> a,
                    const __grid_constant__ StepParams<T> p0, const int* list, int parity, int stage, int pass)
{
    constexpr int LANES = amr_lanes<T>();
    using V = typename ValOf<T, LANES>::V;
    extern __shared__ __align__(16) unsigned char smem_rawq[];
    SmemQ<T, LANES>& s = *reinterpret_cast<SmemQ<T, LANES>*>(smem_rawq);
    __shared__ SubFaces<T> sub;
    const int tid = threadIdx.x;
    const Place<T, LANES> at(tid, blockIdx.x);
    const int ib = list[blockIdx.x];
    const int sc = scen_of(m, ib);
    const StepParams<T>& p = m.sparams ? m.sparams[sc] : p0;
    const int nbm = m.nblkmem, lev = m.level[ib];
    T* const* W = a.W[stage];
    const size_t base = (size_t)ib * 324;
    const bool lead = m.lead ? m.lead[ib] != 0 : pass == 0 && blockIdx.x == 0;
    const bool segs = block_has_segments<T>(m, ib), finer = has_finer_neighbour(m.nbr, nbm, m.level, ib);
    const T delta = calcres<T>(p.delta0, lev);
    // tables alone: ring 1's parent cells (threads 0..63), ring 2's rules (64..127)
    const int sd = (tid >> 4) & 3, t = tid & 15;
    bool coarse = false;
    int pb = 0, px = 0, py = 0;
    CellRule<T> r{};
    if (tid < 64) coarse = parent_cell(m.nbr, nbm, m.level, ib, sd, t, pb, px, py);
    else if (tid < 128) r = outer_rule<T>(m.nbr, nbm, m.level, ib, sd, t);
    BedGradQ<T, LANES> bg;
    load_bedgrad_q<T, ENGINE, LANES>(m, ib, at, bg);
    pdl_wait();
    const V zb = own_of<V>(m.zb + base, hi18(at.x, at.r), 8 * 18, at.l);
    V c[4];
#pragma unroll
    for (int v = 0; v < 4; v++) c[v] = own_of<V>(W[v] + base, hi18(at.x, at.r), 8 * 18, at.l);
    int rx = 0, ry = 0;
    if (tid < 64) {
        // ring 1 (the block's halo, corners excluded) and the coarse/fine substitution
        int hx, hy;
        halo_xy(sd, t, hx, hy);
        const size_t c18 = base + hi18(hx, hy);
#pragma unroll
        for (int v = 0; v < 4; v++) BGF_ROW(s.t[v], pt, hx, hy) = W[v][c18];
        BGF_ROW(s.zb, pz, hx, hy) = m.zb[c18];
        if (t == 0) sub.on[sd] = coarse ? 1 : 0;
        if (coarse) {
            sub.h[sd][t] = W[0][(size_t)pb * 324 + hi18(px, py)];
            sub.z[sd][t] = a.zb[(size_t)pb * 324 + hi18(px, py)];
        }
    } else if (tid < 128) {
        // ring 2: the outer stencil values of the halo gradients
        halo_xy(sd, t, rx, ry);
        if (sd == 0) rx = -2;
        else if (sd == 1) rx = BW + 1;
        else if (sd == 2) ry = -2;
        else ry = BW + 1;
        if (r.kind == 3) {
            // inside a coarser neighbour's 2x2 patch, which may reach into its halo:
            // that neighbour has a finer neighbour, so it runs this chain and its
            // stage tile is filled
#pragma unroll
            for (int v = 0; v < 4; v++) BGF_ROW(s.t[v], pt, rx, ry) = rule_eval(r, Acc324<T>{W[v]});
        }
    }
    const TimeState ts = m.time[2 * sc + parity];
    if (!step_live(ts)) {
        if (stage == 1 && lead && tid == 0) {
            TimeState nt = ts;
            nt.done = 1;
            m.time[2 * sc + (parity ^ 1)] = nt;
        }
        return;
    }
    if (tid >= 64 && tid < 128 && r.kind != 3) {
        // ring 2 at interior cells of this block or of a same-level or finer
        // neighbour, read as the stage reads any cell (the neighbour may run the
        // single-level kernels and have no stage tile): the state of the step
        const T halfdt = stage == 0 ? (T)0 : step_dt<T>(ts, m.dtmin[2 * sc + parity]) * (T)0.5;
        const StageState<T> S{m, p, ts.cur, stage != 0, halfdt, ts.totaltime};
        T cv[4][4];  // per rule cell: h, zs, u, v
        const int nc = r.kind == 0 ? 1 : 4;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (q < nc) {
                S.get(r.b[q], r.x[q], r.y[q], cv[q][0], cv[q][2], cv[q][3]);
                cv[q][1] = a.zb[(size_t)r.b[q] * 324 + hi18(r.x[q], r.y[q])] + cv[q][0];
            }
#pragma unroll
        for (int v = 0; v < 4; v++)
            BGF_ROW(s.t[v], pt, rx, ry) = r.kind == 0 ? cv[0][v] : (T)0.25 * (cv[0][v] + cv[1][v] + cv[2][v] + cv[3][v]);
    }
    if (stage == 1 && tid == 0) {
        const T dt0 = step_dt<T>(ts, m.dtmin[2 * sc + parity]);
        s.dtv = dt0;
        if (p.has_rain && !p.rain_map) {
            // uniform rain (AddrainforcingImplicitCPU): the step's depth, the same for every cell
            const T rr = (T)series_at(m.rain_t + p.rain_off, m.rain_r + p.rain_off, p.rain_n, ts.totaltime,
                                      p.rain_sorted != 0);
            s.rainv = M<T>::fmax_(rr / (T)1000.0 / (T)3600.0 * dt0, (T)0.0);
        }
    }
    store_own<T, LANES>(s, at, c, zb);
    __syncthreads();
    const bool all = segs || finer;
    OwnFlux<V> own;
    T amax = tile_faces<T, ENGINE, LANES, false, true, true>(s, p, delta, at, c, zb, bg, true, own, (T)0, &sub);
    if (stage == 0) warp_max<T, LANES>(s, tid, finite_speed(c[VH], c[VU], c[VV], amax));
    pdl_trigger();
    __syncthreads();  // every face written
    if (pass == 0 && tid < 64) {
        // the faces of a side with a coarser neighbour, at the places of fxi / fyi
        const int n1 = m.nbr[(2 * sd) * nbm + ib], n2 = m.nbr[(2 * sd + 1) * nbm + ib];
        if (m.level[n1] < lev || m.level[n2] < lev) {
            const size_t fb = (size_t)ib * NFX;
            if (sd < 2) {
                const int fx = sd == 0 ? 0 : BW;
                a.F[0][fb + fxi(fx, t)] = BGF_ROW(s.fx[0], pfx, fx, t);
                a.F[1][fb + fxi(fx, t)] = BGF_ROW(s.fxq(), pfx, fx, t);
                a.F[2][fb + fxi(fx, t)] = BGF_ROW(s.fx[1], pfx, fx, t);
                a.F[3][fb + fxi(fx, t)] = BGF_ROW(s.fx[2], pfx, fx, t);
            } else {
                const int fy = sd == 2 ? 0 : BW;
                a.F[4][fb + fyi(t, fy)] = BGF_ROW(s.fy[0], pfy, t, fy);
                a.F[5][fb + fyi(t, fy)] = BGF_ROW(s.fyq(), pfy, t, fy);
                a.F[6][fb + fyi(t, fy)] = BGF_ROW(s.fy[1], pfy, t, fy);
                a.F[7][fb + fyi(t, fy)] = BGF_ROW(s.fy[2], pfy, t, fy);
            }
        }
    }
    if (pass == 0 && finer) return;
    if (stage == 0 && tid == 0) block_dt<T, LANES>(s, p, delta, &m.dtmin[2 * sc + parity]);
    const T dt = stage == 0 ? (T)0 : s.dtv;
    const double dtd = (double)dt;
    const size_t g = (size_t)ib * 256 + at.r * 16 + at.x;
    if (finer) {
        __syncthreads();  // (a side's own faces have been read)
        // HaloFluxCPULR / HaloFluxCPUBT (src/Halo.cu:1441-1540, 1766-1850): the faces of
        // a side with finer neighbours take the mean of the two fine faces
        if (tid < 64) {
            const int nbh = m.nbr[(2 * sd + (t >= BW / 2 ? 1 : 0)) * nbm + ib];
            if (m.level[nbh] > lev) {
                const int jj = t < BW / 2 ? 2 * t : (t - BW / 2) * 2;
                const size_t nf = (size_t)nbh * NFX;
                int f0, f1;
                if (sd == 0) { f0 = fxi(BW, jj); f1 = fxi(BW, jj + 1); }
                else if (sd == 1) { f0 = fxi(0, jj); f1 = fxi(0, jj + 1); }
                else if (sd == 2) { f0 = fyi(jj, BW); f1 = fyi(jj + 1, BW); }
                else { f0 = fyi(jj, 0); f1 = fyi(jj + 1, 0); }
                T* const* F = a.F + (sd < 2 ? 0 : 4);
                auto mean = [&](int q) { return (T)0.5 * (F[q][nf + f0] + F[q][nf + f1]); };
                if (sd < 2) {
                    const int fx = sd == 0 ? 0 : BW;
                    BGF_ROW(s.fx[0], pfx, fx, t) = mean(0);
                    BGF_ROW(s.fxq(), pfx, fx, t) = mean(1);
                    BGF_ROW(s.fx[1], pfx, fx, t) = mean(2);
                    BGF_ROW(s.fx[2], pfx, fx, t) = mean(3);
                } else {
                    const int fy = sd == 2 ? 0 : BW;
                    BGF_ROW(s.fy[0], pfy, t, fy) = mean(0);
                    BGF_ROW(s.fyq(), pfy, t, fy) = mean(1);
                    BGF_ROW(s.fy[1], pfy, t, fy) = mean(2);
                    BGF_ROW(s.fy[2], pfy, t, fy) = mean(3);
                }
            }
        }
    }
    if (segs) {
        // the segments read state n's depth: in the corrector it takes the tile's place
        if (stage == 1) {
            __syncthreads();
            s.t[VH].put(pt(at.x, at.r), at.l, own_of<V>(a.W[0][0] + base, hi18(at.x, at.r), 8 * 18, at.l));
            if (tid < 64) {
                int hx, hy;
                halo_xy(sd, t, hx, hy);
                BGF_ROW(s.t[VH], pt, hx, hy) = a.W[0][0][base + hi18(hx, hy)];
            }
        }
        __syncthreads();
        boundaries_q<T, false, LANES>(s, m, p, ib, stage == 0 ? ts.totaltime + ts.dt * 0.5 : ts.totaltime + dtd, tid,
                                      m.u[ts.cur], m.v[ts.cur]);
    }
    if (all) {
        __syncthreads();
        reload_faces<T, LANES>(s, at, own);
    }
    V dh, dhu, dhv;
    divergence_q<T, LANES>(s, p, (T)1.0 / ((T)1.0 * delta), at, own, c[VH], c[VU], c[VV], dh, dhu, dhv);
    if (stage == 0) {
        // predictor: the tendencies (before the river source), from which the
        // corrector rebuilds the half-step state of any cell (StageState)
        put_own(m.dh, g, at.l, dh);
        put_own(m.dhu, g, at.l, dhu);
        put_own(m.dhv, g, at.l, dhv);
        return;
    }
    if (p.nriver > 0) {
        const int y = at.r + 8 * at.l;
        if constexpr (LANES == 1) dh = add_rivers_q<T>(m, p, ib, at.x, y, dh, ts.totaltime);
        else dh = V{add_rivers_q<T>(m, p, ib, at.x, y, dh.a, ts.totaltime), add_rivers_q<T>(m, p, ib, at.x, y + 8, dh.b, ts.totaltime)};
    }
    const V hold = own_of<V>(m.h[ts.cur], g, 128, at.l), uold = own_of<V>(m.u[ts.cur], g, 128, at.l),
            vold = own_of<V>(m.v[ts.cur], g, 128, at.l);
    const int nxt = ts.cur ^ 1;
    full_step<T, false, LANES, true>(m, p, ib, at, g, nxt, dt, delta, (T)0, s.rainv, ts.totaltime, hold, uold, vold, dh, dhu, dhv);
    if (lead && tid == 0) m.time[2 * sc + (parity ^ 1)] = next_time_state<T>(ts, p, dtd, nxt, m.dtmin + 2 * sc, parity);
}

// ---------------------------------------------------------------- bed preparation

// fillHaloC on the bed (src/Halo.cu:16-51): halo from the neighbours' interiors.
template <class T> __global__ void __launch_bounds__(64) bed_halo_kernel(DevModel<T> m, T* zb)
{
    const int ib = m.active[blockIdx.x];
    const int s = threadIdx.x >> 4, j = threadIdx.x & 15;
    const CellRule<T> r = halo_rule<T>(m.nbr, m.nblkmem, m.level, ib, s, j);
    int hx, hy;
    halo_xy(s, j, hx, hy);
    zb[(size_t)ib * 324 + hi18(hx, hy)] = rule_eval(r, Acc324<T>{zb});
}

// gradientC on the bed (src/Gradients.cu:921-957)
template <class T>
__global__ void __launch_bounds__(NTHREADS) bed_grad_kernel(DevModel<T> m, StepParams<T> p, const T* zb, T* gx, T* gy)
{
    const int ib = m.active[blockIdx.x];
    const int tid = threadIdx.x, x = tid & 15, y = tid >> 4;
    const size_t i = (size_t)ib * 324 + hi18(x, y);
    const T delta = calcres<T>(p.delta0, m.level[ib]);
    const T rdelta = (T)1.0 / delta;
    gx[i] = div_by(minmod2(p.theta, zb[i - 1], zb[i], zb[i + 1]), delta, rdelta);
    gy[i] = div_by(minmod2(p.theta, zb[i - 18], zb[i], zb[i + 18]), delta, rdelta);
}

// gradientHalo on the bed (src/Gradients.cu:2584-2605, 2713-3290)
template <class T>
__global__ void __launch_bounds__(64) bed_grad_halo_kernel(DevModel<T> m, StepParams<T> p, const T* zb, T* gx, T* gy)
{
    const int ib = m.active[blockIdx.x];
    const int s = threadIdx.x >> 4, t = threadIdx.x & 15;
    const T delta = calcres<T>(p.delta0, m.level[ib]);
    const T rdelta = (T)1.0 / delta;
    const T outer = rule_eval(outer_rule<T>(m.nbr, m.nblkmem, m.level, ib, s, t), Acc324<T>{zb});
    const Acc324<T> z{zb};
    int hx, hy;
    halo_xy(s, t, hx, hy);
    const size_t i = (size_t)ib * 324 + hi18(hx, hy);
    if (s == 0) gx[i] = div_by(minmod2(p.theta, outer, zb[i], z(ib, 0, t)), delta, rdelta);
    else if (s == 1) gx[i] = div_by(minmod2(p.theta, z(ib, BW - 1, t), zb[i], outer), delta, rdelta);
    else if (s == 2) gy[i] = div_by(minmod2(p.theta, outer, zb[i], z(ib, t, 0)), delta, rdelta);
    else gy[i] = div_by(minmod2(p.theta, z(ib, t, BW - 1), zb[i], outer), delta, rdelta);
}

// refine_linear on the bed (src/Halo.cu:1044-1394)
template <class T>
__global__ void __launch_bounds__(64) bed_refine_kernel(DevModel<T> m, StepParams<T> p, T* zb, const T* gx, const T* gy)
{
    const int ib = m.active[blockIdx.x];
    const int s = threadIdx.x >> 4, j = threadIdx.x & 15;
    int pb, px, py;
    if (!parent_cell(m.nbr, m.nblkmem, m.level, ib, s, j, pb, px, py)) return;
    int hx, hy;
    halo_xy(s, j, hx, hy);
    zb[(size_t)ib * 324 + hi18(hx, hy)] = refine_value<T>(Acc324<T>{zb}, Acc324<T>{gx}, Acc324<T>{gy}, s, j, pb, px, py,
                                                           m.level[ib], p.delta0, p.delta0_d);
}

// ---------------------------------------------------------------- launchers

template <class T, int ENGINE> static cudaError_t amr_configure_engine()
{
    return cudaFuncSetAttribute(amr_step_kernel<T, ENGINE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(SmemQ<T, amr_lanes<T>()>));
}

template <class T> cudaError_t configure_amr_kernels()
{
    cudaError_t e = amr_configure_engine<T, 1>();
    if (e != cudaSuccess) return e;
    return amr_configure_engine<T, 2>();
}

// A launch that may start while the kernel before it still runs (pdl_wait in the kernel);
// chained = false: a plain launch.
template <class... P, class... A>
static void chain_launch(bool chained, void (*k)(P...), int grid, int nt, size_t smem, cudaStream_t st, const A&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chained ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, k, args...);  // (an error stays for the caller's cudaGetLastError)
}

template <class T>
int launch_amr_stage(const DevModel<T>& m, const AmrDev<T>& a, const StepParams<T>& p, int engine, int parity, int stage,
                     const AmrLists& L, cudaStream_t st)
{
    const int n = m.nblk;
    int launches = 1;
    // (the first launch follows the join with the single-level kernels' branch)
    chain_launch(false, amr_halo_kernel<T>, n, HALO_THREADS, 0, st, m, a, p, parity, stage);
    auto ctas = [](int k) { return (k + SIDE_BLOCKS - 1) / SIDE_BLOCKS; };
    const int nt = 64 * SIDE_BLOCKS, nc = L.coarse_off[L.nlev];
    if (nc) {
        chain_launch(true, amr_refine_kernel<T>, ctas(nc), nt, 0, st, m, a, p, L.coarse, nc, parity, stage);
        launches++;
        if (a.wetdryfix) {
            for (int l = 0; l < L.nlev; l++) {  // coarsest first
                const int k = L.coarse_off[l + 1] - L.coarse_off[l];
                if (!k) continue;
                chain_launch(true, amr_wetdry_kernel<T>, ctas(k), nt, 0, st, m, a, p, L.coarse + L.coarse_off[l], k, parity, stage);
                launches++;
            }
        }
        chain_launch(true, amr_apply_kernel<T>, ctas(nc), nt, 0, st, m, a, L.coarse, nc, parity, stage);
        launches++;
    }
    auto step = engine == 1 ? amr_step_kernel<T, 1> : amr_step_kernel<T, 2>;
    for (int pass = 0; pass < 2; pass++) {
        const int k = pass ? n - L.nofiner : L.ncoarser;
        if (!k) continue;
        chain_launch(true, step, k, Quad<T, amr_lanes<T>()>::NT, sizeof(SmemQ<T, amr_lanes<T>()>), st, m, a, p,
                     m.active + (pass ? L.nofiner : 0), parity, stage, pass);
        launches++;
    }
    return launches;
}

template <class T>
int launch_bed_init(const DevModel<T>& m, const StepParams<T>& p, T* zb, T* gx, T* gy, cudaStream_t st)
{
    const int n = m.nblk;
    bed_halo_kernel<T><<<n, 64, 0, st>>>(m, zb);
    bed_grad_kernel<T><<<n, NTHREADS, 0, st>>>(m, p, zb, gx, gy);
    bed_grad_halo_kernel<T><<<n, 64, 0, st>>>(m, p, zb, gx, gy);
    bed_refine_kernel<T><<<n, 64, 0, st>>>(m, p, zb, gx, gy);
    bed_grad_halo_kernel<T><<<n, 64, 0, st>>>(m, p, zb, gx, gy);
    return 5;
}

template cudaError_t configure_amr_kernels<float>();
template cudaError_t configure_amr_kernels<double>();
template int launch_amr_stage<float>(const DevModel<float>&, const AmrDev<float>&, const StepParams<float>&, int, int,
                                     int, const AmrLists&, cudaStream_t);
template int launch_amr_stage<double>(const DevModel<double>&, const AmrDev<double>&, const StepParams<double>&, int,
                                      int, int, const AmrLists&, cudaStream_t);
template int launch_bed_init<float>(const DevModel<float>&, const StepParams<float>&, float*, float*, float*,
                                    cudaStream_t);
template int launch_bed_init<double>(const DevModel<double>&, const StepParams<double>&, double*, double*, double*,
                                     cudaStream_t);

}  // namespace BGF_VARIANT
}  // namespace bgf
