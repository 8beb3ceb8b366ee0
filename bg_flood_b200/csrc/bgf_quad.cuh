// Single-level stage kernels: pairs of cells eight rows apart.
//
// Same step as flux_kernel / update_kernel (bgf_flow.cuh): the predictor assembles
// the block's 20x20 tile (block + two-cell ring from the neighbour tables), computes
// limited gradients, the wet-slope reset, every X and Y face, the CFL minimum, the
// boundary segments and the flux divergence; the corrector rebuilds the half-step
// tile, repeats the faces and applies the full-step advance, friction and rain.
//
// How the work maps onto the SM (these kernels are bound by instruction issue, not by
// memory, so the layout is the one that needs the fewest instructions per cell):
//
//  * Cells (x, r) and (x, r + 8), r = 0..7, form a pair.  The neighbours of a pair in x and
//    in y are pairs of the same kind.  With LANES = 2 (128 threads per block) a thread owns
//    a pair as one pair value (bgf_pair.cuh): every stencil operand is one 64-bit shared
//    word and every sum and product of both cells one paired instruction, and no registers
//    are moved to form pairs of neighbours.  With LANES = 1 (256 threads) a thread owns one
//    cell of a pair and all values are scalars: twice the warps, each with half the serial
//    work, for FP64 (whose pairs are two scalar streams anyway and take 168 registers) and
//    for meshes with few blocks in the exact build, whose divisions are long chains.  The
//    rule and its figures are beside the launch (bgf_flow.cu).
//  * The shared tile keeps pair rows -2..9; rows 7 and 8 of the block lie in it twice,
//    beside the ring.
//  * A cell's state reconstructed on its two faces of a direction (depth, surface,
//    velocities) is formed once, at the cell: the low side stays in registers for the
//    cell's own face, the high side goes to shared memory for the next cell's face.
//    The quotient of the velocity reconstruction is one per cell and direction.
//  * The faces give the largest wave speed; one division per block turns the largest of
//    all into the block's dt (division is monotonic, so the value is the one that the
//    smallest of the cells' dt has).
//  * The block's extra work (the slopes of the ring, the faces on the right column and
//    the top row) is one pass each of 64 and 32 cells, on different warps chosen by the
//    block's number, so that no scheduler gets it in every resident block (the ring of the
//    exact build's pairs: RingPass).
//
// The exact build evaluates each value with the operations of the one-cell kernels in
// their order and is bit-identical to them.
//
// Measured against the kernels this replaced (pairs of adjacent rows, faces from gradients)
// on B200: 545 -> 525 warp-instructions x 32 per cell in the predictor and 633 -> 635 in the
// corrector (fast FP32); with even shares of the work and the chained launches (pdl_trigger) the step of the 1024x1024
// run-up takes 51.8 instead of 56.6 us, of a 4096x4096 one 729 instead of 769 us.  Two
// pairs per thread (398 and 503 instructions per cell, 128 registers) ran as fast on large
// grids and slower on all others; one warp marching over a block's rows (no barriers) was
// half as fast, its warps out of step in the instruction cache.
//
// Included inside namespace bgf::BGF_VARIANT after bgf_stage.cuh and bgf_pair.cuh.
#pragma once

template <class T, int LANES> struct ValOf {
    using V = V2<T>;
};
template <class T> struct ValOf<T, 1> {
    using V = T;
};

// Threads per block and resident CTAs per SM (launch bounds).
template <class T, int LANES> struct Quad {
    static constexpr int NT = 256 / LANES, NW = NT / 32;
    static constexpr int ctas = sizeof(T) == 8 ? 3 : LANES == 2 ? 7 : 5;
};

// ---------------------------------------------------------------- layouts
// Index of the pair at (x, pair row r).
__device__ __forceinline__ int pt(int x, int r) { return (r + 2) * 20 + x + 2; }  // tile, r = -2..9, x = -2..17
__device__ __forceinline__ int pz(int x, int r) { return (r + 1) * 18 + x + 1; }  // bed, r = -1..8, x = -1..16
__device__ __forceinline__ int pnx(int x, int r) { return r * 17 + x + 1; }       // high X side, x = -1..15
__device__ __forceinline__ int pny(int x, int r) { return (r + 1) * 16 + x; }     // high Y side, r = -1..7
__device__ __forceinline__ int pfx(int x, int r) { return r * 17 + x; }           // X faces, x = 0..16
__device__ __forceinline__ int pfy(int x, int r) { return r * 16 + x; }           // Y faces, r = 0..8

// N pairs of values.  LANES = 2: the two of a pair side by side; LANES = 1: two planes.
template <class T, int N, int LANES> struct Cells {
    using V = typename ValOf<T, LANES>::V;
    T a[2 * N];
    __device__ __forceinline__ T& cell(int p, int l) { return a[LANES == 2 ? 2 * p + l : l * N + p]; }
    __device__ __forceinline__ V get(int p, int l) const
    {
        if constexpr (LANES == 1) {
            return a[l * N + p];
        } else if constexpr (sizeof(T) == 4) {
            const float2 v = *reinterpret_cast<const float2*>(a + 2 * p);
            return V{v.x, v.y};
        } else {
            const double2 v = *reinterpret_cast<const double2*>(a + 2 * p);
            return V{v.x, v.y};
        }
    }
    __device__ __forceinline__ void put(int p, int l, V v)
    {
        if constexpr (LANES == 1) a[l * N + p] = v;
        else if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(a + 2 * p) = make_float2(v.a, v.b);
        else *reinterpret_cast<double2*>(a + 2 * p) = make_double2(v.a, v.b);
    }
};
// The cell of row y of an array indexed by f (rows 8 and beyond: lane 1 of the pair row y - 8).
#define BGF_ROW(arr, f, x, y) arr.cell(f(x, (y) < 8 ? (y) : (y) - 8), (y) < 8 ? 0 : 1)

template <class T, int LANES> struct SmemQ {
    Cells<T, 240, LANES> t[4];   // h, zs, u, v
    Cells<T, 180, LANES> zb;     // bed (split precision: its deviation zb + D)
    Cells<T, 136, LANES> nx[4];  // high X side of each cell: depth, surface (engine 2: bed), u, v
    Cells<T, 144, LANES> ny[4];  // high Y side: depth, surface (bed), v, u; pair row -1 holds rows -1 and 7
    Cells<T, 8, LANES> ex[4];    // low X side of the column x = 16
    T ey[4][16];                 // low Y side of the row y = 16
    Cells<T, 136, LANES> fx[3];  // X faces: Fhu, Su, Fqvx
    Cells<T, 144, LANES> fy[3];  // Y faces: Fhv, Sv, Fquy; pair row 8 holds the faces 8 and 16
    T red[8];
    T dtv;                       // dt of the step (corrector), evaluated once per block
    T rainv;                     // uniform rain depth of the step (corrector)
    // momentum fluxes Fqux and Fqvy, which other threads read only in blocks with boundary
    // segments (and on level interfaces): in place of the tile's u and v, which no face reads
    __device__ __forceinline__ Cells<T, 240, LANES>& fxq() { return t[VU]; }
    __device__ __forceinline__ Cells<T, 240, LANES>& fyq() { return t[VV]; }
};

// The own pair (or cell) of an array of a block: cells g and g + 128 (bed tile: 8 rows of 18).
template <class V, class P> __device__ __forceinline__ V own_of(const P* a, size_t g, int step, int l)
{
    if constexpr (sizeof(V) == sizeof(typename LaneOf<V>::T)) return (V)a[g + step * l];
    else return V{(typename LaneOf<V>::T)a[g], (typename LaneOf<V>::T)a[g + step]};
}
template <class T> __device__ __forceinline__ void put_own(T* a, size_t g, int l, V2<T> v) { a[g] = v.a; a[g + 128] = v.b; }
template <class T> __device__ __forceinline__ void put_own(T* a, size_t g, int l, T v) { a[g + 128 * l] = v; }
// The value of lane 0 or 1, or both.
template <class V, class T> __device__ __forceinline__ V lanes_of(T a, T b, int l)
{
    if constexpr (sizeof(V) == sizeof(T)) return l ? b : a;
    else return V{a, b};
}
template <class T> __device__ __forceinline__ T lane_of(V2<T> v, int l) { return l ? v.b : v.a; }
template <class T> __device__ __forceinline__ T lane_of(T v, int) { return v; }

// ---------------------------------------------------------------- numerics
// Each restates the scalar routine of bgf_numerics.cuh operation by operation.

template <class V> __device__ __forceinline__ V cst(typename LaneOf<V>::T x)
{
    if constexpr (sizeof(V) == sizeof(typename LaneOf<V>::T)) return x;
    else return V{x, x};
}

// minmod2 (src/Util_CPU.cu:243-263).  In the increasing case all three candidates
// are >= +0 and the routine returns their minimum; in the decreasing case all are
// <= -0 and it returns their maximum.
template <class V> __device__ __forceinline__ V minmod_v(V theta, V s0, V s1, V s2)
{
    using T = typename LaneOf<V>::T;
    const auto inc = lt(s0, s1) && lt(s1, s2);
    const auto dec = gt(s0, s1) && gt(s1, s2);
    const V d1 = mul(theta, sub(s1, s0));
    const V d2 = mul(sub(s2, s0), cst<V>((T)0.5));
    const V d3 = mul(theta, sub(s2, s1));
    const V lo = vmin(sel(lt(d2, d1), d2, d1), d3);
    const V hi = vmax(sel(gt(d2, d1), d2, d1), d3);
    return sel(inc, lo, sel(dec, hi, cst<V>((T)0.0)));
}

// x / delta for the block spacing (div_by): the fast build multiplies by the rounded
// reciprocal, the exact build takes Markstein's correctly rounded quotient.
template <class T> __device__ __forceinline__ T divd_v(T x, T d, T r)
{
#if BGF_FAST
    return mul_apart(x, r);
#else
    return div_by<T>(x, d, r);
#endif
}
template <class T> __device__ __forceinline__ V2<T> divd_v(V2<T> x, T d, T r)
{
#if BGF_FAST
    return mul(x, V2<T>{r, r});
#else
    return V2<T>{div_by<T>(x.a, d, r), div_by<T>(x.b, d, r)};
#endif
}

#if BGF_FAST
// min of magnitudes with the product's sign (one instruction)
__device__ __forceinline__ float xmin(float x, float y)
{
    float r;
    asm("min.ftz.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ V2<float> xmin(V2<float> x, V2<float> y) { return V2<float>{xmin(x.a, y.a), xmin(x.b, y.b)}; }
#endif

// Limited slope minmod2(theta, s0, s1, s2) / delta.  Fast FP32 build: s0 < s1 < s2 (or
// s0 > s1 > s2) holds exactly when the product of the one-sided differences is positive (a
// product flushed to zero only drops a slope below 1e-19); the result is then the smaller
// magnitude of theta / delta times the smaller difference and half the central difference
// over delta, with the sign of the latter.  (The bits of the form with three candidates:
// rounding is monotonic.)
template <class V>
__device__ __forceinline__ V slope_q(V th, V thr, V hr, V s0, V s1, V s2, typename LaneOf<V>::T delta,
                                     typename LaneOf<V>::T rdelta)
{
    using T = typename LaneOf<V>::T;
#if BGF_FAST
    if constexpr (sizeof(T) == 4) {
        const V a = sub(s1, s0), b = sub(s2, s1), zero = cst<V>((T)0.0);
        const V p = sel(gt(mul(a, b), zero), xmin(a, b), zero);
        return xmin(mul(thr, p), mul(hr, sub(s2, s0)));
    }
#endif
    (void)thr;
    (void)hr;
    return divd_v(minmod_v<V>(th, s0, s1, s2), delta, rdelta);
}

// Wet-slope reset (wetslope)
template <class V>
__device__ __forceinline__ V wetslope_v(V hdelta, V zsi, V hi, V zsm, V zsp, V dzs, V dh, V dzb)
{
    using T = typename LaneOf<V>::T;
    const V base = sub(zsi, hi);
    const V ddz = sub(dzs, dh);
    const V mzs = mad(mul(cst<V>((T)-1.0), hdelta), ddz, base);  // base - hdelta (dzs - dh)
    const V pzs = mad(hdelta, ddz, base);
    const auto reset = gt(mul(dzs, dzs), mul(dzb, dzb)) && (gt(mzs, zsm) || gt(pzs, zsp));
    return sel(reset, add(dh, dzb), dzs);
}

// A face between cell n (low side) and cell i: the states reconstructed on it (depth,
// surface (engine 2: bed), normal and tangential velocity), the cells' own depths and the
// depth and bed of the source terms (the cells' own, or a coarser cell's at its face).
// Split precision: depths are deviations from the block's datum.
template <class V> struct FaceQ {
    V hI, eI, nI, tI, hN, eN, nN, tN;
    V hi, hn, hsi, hsn, zri, zrn;
};
template <class V> struct FluxQ {
    V Fh, Fq, S, Ft, a;  // a: the face's largest wave speed, 0 where it sets no dt
    typename LaneOf<V>::Mask wet;
};

// face_flux (bgf_numerics.cuh) from the reconstructed states.  Wherever a product feeds a
// sum it is written as mad: the fast build fuses the two, and left to itself the compiler
// does not choose the same product in the scalar and in the paired form.  A face that one
// block solves as a scalar (the right column and the top row) is half of a pair on its
// neighbour, and has to come out the same on both (mass is conserved to rounding then).
template <class V, int ENGINE>
__device__ __forceinline__ FluxQ<V> face_q(const FaceQ<V>& f, V g, V ga, V epsi, V eps)
{
    using T = typename LaneOf<V>::T;
    const V zero = cst<V>((T)0.0), half = cst<V>((T)0.5), two = cst<V>((T)2.0), mone = cst<V>((T)-1.0);
    const V nga = mul(mone, ga);
    FluxQ<V> r;
    r.wet = gt(f.hi, eps) || gt(f.hn, eps);
    V fh, fu, ft, fq, s, a;
    if constexpr (ENGINE == 2) {
        // KurgSolver (src/Kurganov.cu:1865-1911)
        const V zlr = vmax(f.eI, f.eN);
        const V hp = vmax(zero, sub(add(f.hI, f.eI), zlr));
        const V hm = vmax(zero, sub(add(f.hN, f.eN), zlr));
        const V up = f.nI, um = f.nN;
        const V cp = vsqrt(mul(g, hp)), cm = vsqrt(mul(g, hm));
        const V ap = vmax(vmax(add(up, cp), add(um, cm)), zero);
        const V am = vmin(vmin(sub(up, cp), sub(um, cm)), zero);
        a = vmax(ap, mul(mone, am));
        const auto live = gt(a, epsi);
        const V ad = dv(cst<V>((T)1.0), sub(ap, am));
        const V qm = mul(hm, um), qp = mul(hp, up), apm = mul(ap, am);
        const V nam = mul(mone, am);
        const V fhl = mul(mad(apm, sub(hp, hm), mad(ap, qm, mul(nam, qp))), ad);
        const V ful = mul(mad(apm, sub(qp, qm),
                              mad(ap, mad(qm, um, mul(ga, mul(hm, hm))), mul(nam, mad(qp, up, mul(ga, mul(hp, hp)))))),
                          ad);
        fh = sel(live, fhl, zero);
        fu = sel(live, ful, zero);
        a = sel(live, a, zero);
        ft = mul(sel(gt(fh, zero), f.tN, f.tI), fh);
        fq = mad(nga, mad(add(f.hI, f.hsi), sub(f.zri, f.eI), sub_mad(mul(hp, hp), f.hI, f.hI)), fu);
        s = mad(nga, mad(add(f.hN, f.hsn), sub(f.zrn, f.eN), sub_mad(mul(hm, hm), f.hN, f.hN)), fu);
    } else {
        const V zA = vmax(sub(f.eI, f.hI), sub(f.eN, f.hN));
        const V zCN = vmin(zA, vmin(f.eN, f.eI));
        const V hp = vmax(zero, vmin(sub(f.eI, zCN), f.hI));
        const V hm = vmax(zero, vmin(sub(f.eN, zCN), f.hN));
        const V up = f.nI, um = f.nN;
        const V cm = vsqrt(mul(g, hm)), cp = vsqrt(mul(g, hp));
        const V fhm = mul(um, hm), fhp = mul(up, hp);
        // hllc (src/Reimann.cu:838-877)
        const V ustar = sub(mad(add(um, up), half, cm), cp);
        const V cstar = mad(add(cm, cp), half, mul(sub(um, up), cst<V>((T)0.25)));
        const V SL = sel(eq(hm, zero), mad(cst<V>((T)-2.0), cp, up), vmin(sub(um, cm), sub(ustar, cstar)));
        const V SR = sel(eq(hp, zero), mad(two, cm, um), vmax(add(up, cp), add(ustar, cstar)));
        const V fum = mul(hm, mad(um, um, mul(mul(g, hm), half)));
        const V fup = mul(hp, mad(up, up, mul(mul(g, hp), half)));
        const V SLSR = mul(SL, SR);
        const V den = sub(SR, SL);
        const V nSL = mul(mone, SL);
        const V nh = mad(SLSR, sub(hp, hm), mad(nSL, fhp, mul(SR, fhm)));
        const V nq = mad(SLSR, mad_sub(hp, up, fhm), mad(nSL, fup, mul(SR, fum)));
        V fhM, fqM;
#if BGF_FAST
        if constexpr (sizeof(T) == 4) {
            // one reciprocal of the wave-speed spread for both star-region fluxes
            const V rden = rcp_v(den);
            fhM = mul(nh, rden);
            fqM = mul(nq, rden);
        } else
#endif
        {
            fhM = dv(nh, den);
            fqM = dv(nq, den);
        }
        const auto caseL = le(zero, SL);
        const auto caseR = ge(zero, SR);
        fh = sel(caseL, fhm, sel(caseR, fhp, fhM));
        fu = sel(caseL, fum, sel(caseR, fup, fqM));
        a = vmax(vabs(SL), vabs(SR));
        ft = mul(sel(gt(fh, zero), f.tN, f.tI), fh);
        fq = mad(mul(nga, add(f.hsi, hp)), sub(f.zri, zCN), fu);
        s = mad(mul(nga, add(hm, f.hsn)), sub(f.zrn, zCN), fu);
    }
    r.Fh = sel(r.wet, fh, zero);
    r.Fq = sel(r.wet, fq, zero);
    r.S = sel(r.wet, s, zero);
    r.Ft = sel(r.wet, ft, zero);
    r.a = sel(r.wet && gt(a, epsi), a, zero);
    return r;
}

// face_flux_split (bgf_split.cuh) from the reconstructed states: momentum fluxes carry
// the datum's hydrostatic shift -g D^2 / 2, which a dry face carries alone.  zri, zrn:
// beds as deviations zb + D (engine 2: zs - h').
template <class V, int ENGINE>
__device__ __forceinline__ FluxQ<V> face_q_split(const FaceQ<V>& f, V D, V g, V ga, V epsi, V eps)
{
    using T = typename LaneOf<V>::T;
    const V zero = cst<V>((T)0.0), one = cst<V>((T)1.0), two = cst<V>((T)2.0), mone = cst<V>((T)-1.0);
    const V half = cst<V>((T)0.5), quarter = cst<V>((T)0.25);
    const V nD = mul(mone, D), nga = mul(mone, ga);
    const V shift = mul(mul(nga, D), D);  // -ga * D * D
    FluxQ<V> r;
    const V Hi = add(D, f.hi), Hn = add(D, f.hn);  // full depths
    r.wet = gt(Hi, eps) || gt(Hn, eps);
    V fh, fu, ft, fq, s, a;
    if constexpr (ENGINE == 2) {
        const V zlr = vmax(f.eI, f.eN);
        const V up = f.nI, um = f.nN;
        const V hp = vmax(nD, sub(add(f.hI, f.eI), zlr));
        const V hm = vmax(nD, sub(add(f.hN, f.eN), zlr));
        const V Hp = add(D, hp), Hm = add(D, hm), Hl = add(D, f.hI), Hr = add(D, f.hN);
        const V cp = vsqrt(mul(g, Hp)), cmo = vsqrt(mul(g, Hm));
        const V ap = vmax(vmax(add(up, cp), add(um, cmo)), zero);
        const V am = vmin(vmin(sub(up, cp), sub(um, cmo)), zero);
        a = vmax(ap, mul(mone, am));
        const auto live = gt(a, epsi);
        const V ad = dv(one, sub(ap, am));
        const V qm = mul(Hm, um), qp = mul(Hp, up), apm = mul(ap, am);
        const V pm = mul(mul(ga, hm), mad(two, D, hm)), pp = mul(mul(ga, hp), mad(two, D, hp));
        const V nam = mul(mone, am);
        const V fhl = mul(mad(apm, sub(hp, hm), mad(ap, qm, mul(nam, qp))), ad);
        const V ful = mul(mad(apm, sub(qp, qm), mad(ap, mad(qm, um, pm), mul(nam, mad(qp, up, pp)))), ad);
        fh = sel(live, fhl, zero);
        fu = sel(live, ful, shift);
        a = sel(live, a, zero);
        ft = mul(sel(gt(fh, zero), f.tN, f.tI), fh);
        fq = mad(nga, mad(sub(hp, f.hI), add(Hp, Hl), mul(add(Hl, Hi), sub(f.zri, f.eI))), fu);
        s = mad(nga, mad(sub(hm, f.hN), add(Hm, Hr), mul(add(Hr, Hn), sub(f.zrn, f.eN))), fu);
    } else {
        const V zA = vmax(sub(f.eI, f.hI), sub(f.eN, f.hN));
        const V zCN = vmin(zA, add(vmin(f.eN, f.eI), D));
        const V hCNr = vmax(nD, vmin(sub(f.eI, zCN), f.hI));
        const V hCNl = vmax(nD, vmin(sub(f.eN, zCN), f.hN));
        // hllc on the reconstructed states, pressures shifted by the datum
        const V hm = add(D, hCNl), hp = add(D, hCNr), um = f.nN, up = f.nI;
        const V cmo = vsqrt(mul(g, hm)), cp = vsqrt(mul(g, hp));
        const V ustar = sub(mad(add(um, up), half, cmo), cp);
        const V cstar = mad(add(cmo, cp), half, mul(sub(um, up), quarter));
        const V SL = sel(eq(hm, zero), mad(cst<V>((T)-2.0), cp, up), vmin(sub(um, cmo), sub(ustar, cstar)));
        const V SR = sel(eq(hp, zero), mad(two, cmo, um), vmax(add(up, cp), add(ustar, cstar)));
        const V fum = mad(mul(hm, um), um, mul(mul(ga, hCNl), mad(two, D, hCNl)));
        const V fup = mad(mul(hp, up), up, mul(mul(ga, hCNr), mad(two, D, hCNr)));
        const V fhm = mul(um, hm), fhp = mul(up, hp);
        const V rs = dv(one, sub(SR, SL));
        const V SLSR = mul(SL, SR);
        const V nSL = mul(mone, SL);
        const V fhM = mul(mad(SLSR, sub(hCNr, hCNl), mad(nSL, fhp, mul(SR, fhm))), rs);
        const V fqM = mul(mad(SLSR, sub_apart(mul(hp, up), mul(hm, um)), mad(nSL, fup, mul(SR, fum))), rs);
        const auto caseL = le(zero, SL);
        const auto caseR = ge(zero, SR);
        fh = sel(caseL, fhm, sel(caseR, fhp, fhM));
        fu = sel(caseL, fum, sel(caseR, fup, fqM));
        a = vmax(vabs(SL), vabs(SR));
        ft = mul(sel(gt(fh, zero), f.tN, f.tI), fh);
        fq = mad(mul(nga, add(Hi, add(D, hCNr))), sub(f.zri, zCN), fu);
        s = mad(mul(nga, add(add(D, hCNl), Hn)), sub(f.zrn, zCN), fu);
    }
    r.Fh = sel(r.wet, fh, zero);
    r.Fq = sel(r.wet, fq, shift);
    r.S = sel(r.wet, s, shift);
    r.Ft = sel(r.wet, ft, zero);
    r.a = sel(r.wet && gt(a, epsi), a, zero);
    return r;
}

// AdvkernelCPU / AdvkernelGPU (src/Advection.cu:272-385) per lane.
template <class T>
__device__ __forceinline__ T edt_lane(T dt, double eps_d, bool forcemass, T hold, T dhi)
{
#if BGF_FAST
    return forcemass ? dt : dhi >= (T)0.0 ? dt : M<T>::fmin_(dt, dv(M<T>::fmax_(hold, (T)eps_d), M<T>::fabs_(dhi)));
#else
    return forcemass ? dt : dhi >= (T)0.0 ? dt : (T)fmin((double)dt, fmax((double)hold, eps_d) / (double)M<T>::fabs_(dhi));
#endif
}
template <class T> __device__ __forceinline__ T edt_v(T dt, double eps_d, bool fm, T hold, T dhi)
{
    return edt_lane<T>(dt, eps_d, fm, hold, dhi);
}
template <class T> __device__ __forceinline__ V2<T> edt_v(T dt, double eps_d, bool fm, V2<T> hold, V2<T> dhi)
{
    return V2<T>{edt_lane<T>(dt, eps_d, fm, hold.a, dhi.a), edt_lane<T>(dt, eps_d, fm, hold.b, dhi.b)};
}
template <class V>
__device__ __forceinline__ void advance_v(typename LaneOf<V>::T dt, typename LaneOf<V>::T eps, double eps_d,
                                          bool forcemass, V hold, V uold, V vold, V dhi, V dhui, V dhvi, V& ho, V& uo,
                                          V& vo)
{
    using T = typename LaneOf<V>::T;
    const V edt = edt_v(dt, eps_d, forcemass, hold, dhi);
    ho = mad(edt, dhi, hold);
    const auto wet = gt(ho, cst<V>(eps));
    uo = sel(wet, dv(mad(hold, uold, mul(edt, dhui)), ho), cst<V>((T)0.0));
    vo = sel(wet, dv(mad(hold, vold, mul(edt, dhvi)), ho), cst<V>((T)0.0));
}

// advance_split (bgf_split.cuh): depths as deviations from the datum D, full depths for the
// limiter and the velocities.
template <class T> __device__ __forceinline__ T edt_split(T dt, T eps, bool forcemass, T Hold, T dhi)
{
    return forcemass ? dt : dhi >= (T)0.0 ? dt : M<T>::fmin_(dt, dv(M<T>::fmax_(Hold, eps), M<T>::fabs_(dhi)));
}
template <class T> __device__ __forceinline__ V2<T> edt_split(T dt, T eps, bool forcemass, V2<T> Hold, V2<T> dhi)
{
    return V2<T>{edt_split<T>(dt, eps, forcemass, Hold.a, dhi.a), edt_split<T>(dt, eps, forcemass, Hold.b, dhi.b)};
}
template <class V>
__device__ __forceinline__ void advance_split_v(typename LaneOf<V>::T dt, typename LaneOf<V>::T eps, bool forcemass, V D,
                                                V hold, V uold, V vold, V dhi, V dhui, V dhvi, V& ho, V& uo, V& vo)
{
    using T = typename LaneOf<V>::T;
    const V Hold = add(D, hold);
    const V edt = edt_split(dt, eps, forcemass, Hold, dhi);
    ho = mad(edt, dhi, hold);
    const V Ho = add(D, ho);
    const auto wet = gt(Ho, cst<V>(eps));
    uo = sel(wet, dv(mad(Hold, uold, mul(edt, dhui)), Ho), cst<V>((T)0.0));
    vo = sel(wet, dv(mad(Hold, vold, mul(edt, dhvi)), Ho), cst<V>((T)0.0));
}

// Cube root and smart friction per lane.  (The latter out of line: its logarithm and
// quotients crowd the corrector's instruction cache in the runs that do not use it.)
template <class T> __device__ __forceinline__ T cbrt_v(T h)
{
#if BGF_FAST
    if constexpr (sizeof(T) == 4) return cbrta(h);
#endif
    return M<T>::cbrt_(h);
}
template <class T> __device__ __forceinline__ V2<T> cbrt_v(V2<T> h) { return V2<T>{cbrt_v<T>(h.a), cbrt_v<T>(h.b)}; }
template <class T> __device__ __noinline__ T smartfriction_nl(T hi, T zo) { return smartfriction<T>(hi, zo); }
template <class T> __device__ __forceinline__ T smart_v(T h, T z) { return smartfriction_nl<T>(h, z); }
template <class T> __device__ __forceinline__ V2<T> smart_v(V2<T> h, V2<T> z)
{
    return V2<T>{smartfriction_nl<T>(h.a, z.a), smartfriction_nl<T>(h.b, z.b)};
}

// bottomfriction (src/Friction.cu:17-143); model is uniform.
template <class V>
__device__ __forceinline__ void friction_v(int model, typename LaneOf<V>::T g, typename LaneOf<V>::T eps,
                                           typename LaneOf<V>::T dt, V cfv, V hi, V& ui, V& vi)
{
    using T = typename LaneOf<V>::T;
    const V normu = vsqrt(mad(ui, ui, mul(vi, vi)));
    V cfi;
    if (model == 0) cfi = cfv;
    else if (model == 1) cfi = smart_v(hi, cfv);
    else if (model == -1) cfi = dv(mul(mul(cst<V>(g), cfv), cfv), cbrt_v(hi));
    else cfi = cst<V>((T)0.0);
    const V den = mad(dv(mul(cfi, normu), hi), cst<V>(dt), cst<V>((T)1.0));
    const auto wet = gt(hi, cst<V>(eps));
    ui = sel(wet, dv(ui, den), ui);
    vi = sel(wet, dv(vi, den), vi);
}

// ---------------------------------------------------------------- phases

// The two cells of ring element k (0..63) of a block's tile, as cells k and k + 64: for
// k < 32 the ring columns -1, -2, 16, 17 at rows (k & 7) and (k & 7) + 8, beyond them the
// ring rows (-1, 16) and (-2, 17) at column k & 15.  Gives the cell's tile position and its
// source.
template <class T>
__device__ __forceinline__ void ring_cell(const DevModel<T>& m, int ib, int k, int& x, int& y, int& sb, int& sx, int& sy)
{
    const int second = k >> 6, e = k & 63, d = e < 32 ? (e >> 3) & 1 : (e >> 4) & 1;
    const int side = e < 32 ? e >> 4 : 2 + second;  // left, right, bottom, top
    const int t = e < 32 ? (e & 7) + 8 * second : e & 15;
    const int out = side & 1 ? BW + d : -1 - d;            // position across the side
    const int edge = side & 1 ? BW - 1 : 0, in = side & 1 ? d : BW - 1 - d;
    bool has;
    if (m.regular_nbx > 0) {
        const int nbx = m.regular_nbx, nby = m.regular_nby;
        const int by = m.regular_magic ? (int)__umulhi((unsigned)ib, m.regular_magic) : ib / nbx;
        const int bx = ib - by * nbx;
        has = side == 0 ? bx > 0 : side == 1 ? bx < nbx - 1 : side == 2 ? by > 0 : by < nby - 1;
        sb = has ? ib + (side & 1 ? 1 : -1) * (side < 2 ? 1 : nbx) : ib;
    } else {
        sb = m.nbr[(size_t)(2 * side) * m.nblkmem + ib];
        has = sb != ib;
        // a cross-level side raises the error word and falls back to the block's own edge
        if (has ? m.checklev && m.level[sb] != m.level[ib] : m.nbr[(size_t)(2 * side + 1) * m.nblkmem + ib] != ib) {
            atomicOr(m.err, 1);
            sb = ib;
            has = false;
        }
    }
    const int src = has ? in : edge;
    x = side < 2 ? out : t;
    y = side < 2 ? t : out;
    sx = side < 2 ? src : t;
    sy = side < 2 ? t : src;
}

// Whether the slopes of the ring are spread over threads 0..127 (two a ring cell) instead of
// made by two warps: the exact build's are long enough to
// keep the other warps waiting (12,288 blocks: 426 instead of 453 us per step when this was
// chosen), the fast build's are not (151 instead of 148 us).
template <class T, int LANES> struct RingPass {
#if BGF_FAST
    static constexpr bool spread = false;
#else
    static constexpr bool spread = LANES == 2;
#endif
};

// A thread's place in the block: column, pair row and lane of its cells, and whether its
// warp makes the ring slopes (their lane: rl) or the extra faces.
template <class T, int LANES> struct Place {
    int tid, x, r, l, rl;
    bool ring, extra;
    __device__ __forceinline__ Place(int tid_, int w) : tid(tid_), x(tid_ & 15), r((tid_ >> 4) & 7), l(LANES == 2 ? 0 : tid_ >> 7)
    {
        constexpr int NW = Quad<T, LANES>::NW;
        const int hsh = (int)(((unsigned)w * 0x9E3779B1u) >> 30);
        const int at = ((tid_ >> 5) + hsh) & (NW - 1);
        ring = at == 0 || at == (LANES == 2 ? 1 : 4);
        rl = at != 0;
        extra = at == 2;
    }
};

// Bed gradients the engine-1 wet-slope reset reads: the own ones and those of the thread's
// ring cells (spread: towards the block).
template <class T, int LANES> struct BedGradQ {
    typename ValOf<T, LANES>::V gx, gy;
    T ring;
};
template <class T, int ENGINE, int LANES>
__device__ __forceinline__ void load_bedgrad_q(const DevModel<T>& m, int ib, const Place<T, LANES>& at, BedGradQ<T, LANES>& b)
{
    using V = typename ValOf<T, LANES>::V;
    if constexpr (ENGINE == 1) {
        const T* bx = m.dzbdx + (size_t)ib * 324;
        const T* by = m.dzbdy + (size_t)ib * 324;
        const int c = hi18(at.x, at.r);
        b.gx = own_of<V>(bx, c, 8 * 18, at.l);
        b.gy = own_of<V>(by, c, 8 * 18, at.l);
        if constexpr (RingPass<T, LANES>::spread) {
            const int side = at.tid >> 5, t = (at.tid >> 1) & 15;
            const T q = side < 2 ? bx[hi18(side ? BW : -1, t)] : by[hi18(t, side == 3 ? BW : -1)];
            b.ring = side & 1 ? -q : q;
        } else if (at.ring) {
            const int l = at.tid & 31;
            const T* p = l < 16 ? bx + hi18(l < 8 ? -1 : BW, l & 7) : by + hi18(l & 15, -1);
            b.ring = p[at.rl ? (l < 16 ? 8 : 17) * 18 : 0];
        }
    }
}

// The own cells (state and bed) into the tile, the rows 7 and 8 also beside the ring rows.
template <class T, int LANES, class V>
__device__ __forceinline__ void store_own(SmemQ<T, LANES>& s, const Place<T, LANES>& at, const V (&c)[4], V zb)
{
    const int o = pt(at.x, at.r);
#pragma unroll
    for (int v = 0; v < 4; v++) s.t[v].put(o, at.l, c[v]);
    s.zb.put(pz(at.x, at.r), at.l, zb);
    if (at.r == 0 && (LANES == 2 || at.l == 1)) {
#pragma unroll
        for (int v = 0; v < 4; v++) s.t[v].cell(pt(at.x, 8), 0) = lane_of(c[v], 1);
    }
    if (at.r == 7 && at.l == 0) {
#pragma unroll
        for (int v = 0; v < 4; v++) s.t[v].cell(pt(at.x, -1), 1) = lane_of(c[v], 0);
        s.zb.cell(pz(at.x, -1), 1) = lane_of(zb, 0);
    }
}

// A ring cell into the tile, its bed where the block's own halo has one.
template <class T, int LANES>
__device__ __forceinline__ void store_ring(SmemQ<T, LANES>& s, int x, int y, T h, T u, T v, T z)
{
    BGF_ROW(s.t[VH], pt, x, y) = h;
    BGF_ROW(s.t[VU], pt, x, y) = u;
    BGF_ROW(s.t[VV], pt, x, y) = v;
    BGF_ROW(s.t[VZS], pt, x, y) = z + h;
    if (x >= -1 && x <= BW && y >= -1 && y <= BW) BGF_ROW(s.zb, pz, x, y) = z;
}

// 1 + x / y and 1 - x / y.  Fast FP32 build: the product with the reciprocal fused into the sum.
template <class V> __device__ __forceinline__ void one_pm_quot(V x, V y, V& plus, V& minus)
{
    using T = typename LaneOf<V>::T;
    const V one = cst<V>((T)1.0);
#if BGF_FAST
    if constexpr (sizeof(T) == 4) {
        const V r = rcp_v(y);
        plus = mad(x, r, one);
        minus = mad(mul(cst<V>((T)-1.0), x), r, one);
    } else {
        const V q = dv(x, y);
        plus = add_apart(one, q);
        minus = sub_apart(one, q);
    }
#else
    const V q = dv(x, y);
    plus = add(one, q);
    minus = sub(one, q);
#endif
}

// The two sides of a direction reconstructed from a cell's state and limited slopes:
// depth, surface (engine 2: bed), normal and tangential velocity.  q: the scaled depth
// slope over the depth (engine 1, Bouchut velocity reconstruction), wet: where it applies.
template <class V> struct SideQ {
    V h, e, n, t;
};
template <class V, int ENGINE>
__device__ __forceinline__ void both_sides(V dx, V h, V zs, V un, V ut, V gh, V gz, V gn, V gt_, V Hfull, V epsv,
                                           SideQ<V>& lo, SideQ<V>& hi)
{
    using T = typename LaneOf<V>::T;
    const V ndx = mul(cst<V>((T)-1.0), dx);
    lo.h = mad(ndx, gh, h);
    hi.h = mad(dx, gh, h);
    if constexpr (ENGINE == 1) {
        lo.e = mad(ndx, gz, zs);
        hi.e = mad(dx, gz, zs);
        const auto wet = gt(Hfull, epsv);
        V lowq, highq;
        one_pm_quot<V>(mul(dx, gh), Hfull, lowq, highq);
        const V cl = sel(wet, mul(lowq, ndx), ndx);
        const V ch = sel(wet, mul(highq, dx), dx);
        lo.n = mad(cl, gn, un);
        lo.t = mad(cl, gt_, ut);
        hi.n = mad(ch, gn, un);
        hi.t = mad(ch, gt_, ut);
    } else {
        const V z = sub(zs, h), gb = sub(gz, gh);
        lo.e = mad(ndx, gb, z);
        hi.e = mad(dx, gb, z);
        lo.n = mad(ndx, gn, un);
        lo.t = mad(ndx, gt_, ut);
        hi.n = mad(dx, gn, un);
        hi.t = mad(dx, gt_, ut);
    }
}

// What the faces leave for the divergence: the low X face's mass and momentum and tangential
// flux, the same of the low Y face.
template <class V> struct OwnFlux {
    V xh, xq, xt, yh, yq, yt;
};

// Slopes, reconstructed sides and every face of an assembled tile (one barrier between
// the two halves; the caller puts one before and one after).  SPEED: returns the largest
// wave speed that sets this thread's cells' dt.  SUB: faces on a side whose neighbour is
// coarser take that neighbour's cell (subf) as their source-term depth and bed.  allfaces:
// store the momentum fluxes too.
template <class T, int ENGINE, int LANES, bool SPLIT, bool SPEED, bool SUB, class V>
__device__ __forceinline__ T tile_faces(SmemQ<T, LANES>& s, const StepParams<T>& p, T delta, const Place<T, LANES>& at,
                                        const V (&c)[4], V zb, const BedGradQ<T, LANES>& bg, bool allfaces, OwnFlux<V>& own,
                                        T D = (T)0, const SubFaces<T>* subf = nullptr)
{
    const T rdelta = (T)1.0 / delta, thr_s = p.theta * rdelta, hr_s = (T)0.5 * rdelta, hd_s = delta * (T)0.5;
    const V th = cst<V>(p.theta), thr = cst<V>(thr_s), hr = cst<V>(hr_s), dx = cst<V>(hd_s);
    const V eps = cst<V>(p.epsface), Dv = cst<V>(D);
    const int x = at.x, r = at.r, l = at.l, lane = at.tid & 31, o = pt(x, r);
    auto full = [&](V h) { return SPLIT ? add(Dv, h) : h; };
    const V Hc = full(c[VH]);
    SideQ<V> X, Y;  // low sides
    {
        V gr[4], xm[4], xp[4];
#pragma unroll
        for (int v = 0; v < 4; v++) {
            xm[v] = s.t[v].get(o - 1, l);
            xp[v] = s.t[v].get(o + 1, l);
            gr[v] = slope_q<V>(th, thr, hr, xm[v], c[v], xp[v], delta, rdelta);
        }
        if constexpr (ENGINE == 1) gr[VZS] = wetslope_v<V>(dx, c[VZS], Hc, xm[VZS], xp[VZS], gr[VZS], gr[VH], bg.gx);
        SideQ<V> hi;
        both_sides<V, ENGINE>(dx, c[VH], c[VZS], c[VU], c[VV], gr[VH], gr[VZS], gr[VU], gr[VV], Hc, eps, X, hi);
        const int on = pnx(x, r);
        s.nx[0].put(on, l, hi.h);
        s.nx[1].put(on, l, hi.e);
        s.nx[2].put(on, l, hi.n);
        s.nx[3].put(on, l, hi.t);
    }
    {
        V gr[4], ym[4];
#pragma unroll
        for (int v = 0; v < 4; v++) {
            // (one cell per thread: row 8's lower neighbour is lane 0 of row 7, beside the ring)
            ym[v] = s.t[v].get(o - 20, l);
            gr[v] = slope_q<V>(th, thr, hr, ym[v], c[v], s.t[v].get(o + 20, l), delta, rdelta);
        }
        // (interior rows compare both reconstructions with the lower neighbour, WetsloperesetCPU)
        if constexpr (ENGINE == 1) gr[VZS] = wetslope_v<V>(dx, c[VZS], Hc, ym[VZS], ym[VZS], gr[VZS], gr[VH], bg.gy);
        SideQ<V> hi;
        both_sides<V, ENGINE>(dx, c[VH], c[VZS], c[VV], c[VU], gr[VH], gr[VZS], gr[VV], gr[VU], Hc, eps, Y, hi);
        const int on = pny(x, r);
        s.ny[0].put(on, l, hi.h);
        s.ny[1].put(on, l, hi.e);
        s.ny[2].put(on, l, hi.n);
        s.ny[3].put(on, l, hi.t);
        if (r == 7 && l == 0) {
            const int o1 = pny(x, -1);
            s.ny[0].cell(o1, 1) = lane_of(hi.h, 0);
            s.ny[1].cell(o1, 1) = lane_of(hi.e, 0);
            s.ny[2].cell(o1, 1) = lane_of(hi.n, 0);
            s.ny[3].cell(o1, 1) = lane_of(hi.t, 0);
        }
    }
    // ---- the inward sides of the 64 ring cells: two threads a cell (side tid / 32), one for
    // depth and surface, one for the velocities; slopes towards the block (the two orders of a
    // stencil give opposite signs, exactly).
    if constexpr (RingPass<T, LANES>::spread) {
        const int side = at.tid >> 5, t = (at.tid >> 1) & 15, part = at.tid & 1;
        const int hx = side == 0 ? -1 : side == 1 ? BW : t, hy = side < 2 ? t : side == 2 ? -1 : BW;
        const int pr = pt(hx, hy < 8 ? hy : hy - 8), pl = hy < 8 ? 0 : 1;
        const int i = LANES == 2 ? 2 * pr + pl : pl * 240 + pr;
        const int step = (side < 2 ? 1 : 20) * LANES, in = side & 1 ? -step : step;
        const T* a0 = s.t[part ? (side < 2 ? VU : VV) : VH].a;
        const T* a1 = s.t[part ? (side < 2 ? VV : VU) : VZS].a;
        const T n0 = a0[i], n1 = a1[i], f1 = a1[i - in], i1 = a1[i + in];
        T g0 = slope_q<T>(p.theta, thr_s, hr_s, a0[i - in], n0, a0[i + in], delta, rdelta);
        T g1 = slope_q<T>(p.theta, thr_s, hr_s, f1, n1, i1, delta, rdelta);
        T o0, o1;
        if constexpr (ENGINE == 1) {
            const T Hr = SPLIT ? D + n0 : n0;
            T c1 = hd_s;
            if (part == 0) {
                g1 = wetslope_v<T>(hd_s, n1, Hr, f1, i1, g1, g0, bg.ring);
                // the velocities' factor (both_sides)
                T lowq, highq;
                one_pm_quot<T>(mul(hd_s, g0), Hr, lowq, highq);
                c1 = sel(gt(Hr, p.epsface), mul(highq, hd_s), hd_s);
            }
            c1 = __shfl_sync(0xffffffffu, c1, lane & ~1);
            if (part == 0) c1 = hd_s;
            o0 = mad(c1, g0, n0);
            o1 = mad(c1, g1, n1);
        } else {
            o0 = mad(hd_s, g0, n0);
            o1 = part ? mad(hd_s, g1, n1) : mad(hd_s, sub(g1, g0), sub(n1, n0));
        }
        T* q;
        int nq;
        if (side == 0) { const int k = pnx(-1, t & 7); q = s.nx[0].a + (LANES == 2 ? 2 * k + pl : pl * 136 + k); nq = 272; }
        else if (side == 1) { const int k = t & 7; q = s.ex[0].a + (LANES == 2 ? 2 * k + pl : pl * 8 + k); nq = 16; }
        else if (side == 2) { q = s.ny[0].a + LANES * pny(t, -1); nq = 288; }
        else { q = s.ey[0] + t; nq = 16; }
        q += 2 * part * nq;
        q[0] = o0;
        q[nq] = o1;
    }
    // ---- the ring in two warps (rl): lanes 0..7 the column -1, 8..15 the column 16 (rows
    // 0..7 and 8..15), lanes 16..31 the rows -1 and 16.  The inward side only.
    if (!RingPass<T, LANES>::spread && at.ring) {
        const bool isx = lane < 16;
        // tile index of the cell, step across the side
        const int pa = pt(isx ? (lane < 8 ? -1 : BW) : lane & 15, isx ? lane & 7 : at.rl ? 8 : -1);
        const int ia = LANES == 2 ? 2 * pa + at.rl : 240 * at.rl + pa;
        const int d = (isx ? 1 : 20) * LANES;
        const int iu = isx ? VU : VV, iv = isx ? VV : VU;
        const T sg = (isx ? lane >= 8 : at.rl != 0) ? -hd_s : hd_s;
        T q0[4], gr[4], zm, zp;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const T* a = s.t[j == 0 ? VH : j == 1 ? VZS : j == 2 ? iu : iv].a + ia;
            const T m0 = a[-d], p0 = a[d];
            q0[j] = a[0];
            gr[j] = slope_q<T>(p.theta, thr_s, hr_s, m0, q0[j], p0, delta, rdelta);
            if (j == 1) { zm = m0; zp = p0; }
        }
        const T Hr = SPLIT ? D + q0[0] : q0[0];
        if constexpr (ENGINE == 1) gr[1] = wetslope_v<T>(hd_s, q0[1], Hr, zm, zp, gr[1], gr[0], bg.ring);
        SideQ<T> in, outw;
        // (both_sides with the signed half spacing: its high side is the inward one)
        both_sides<T, ENGINE>(sg, q0[0], q0[1], q0[2], q0[3], gr[0], gr[1], gr[2], gr[3], Hr, p.epsface, outw, in);
        T* da;
        int na;  // step between the values' arrays
        if (lane < 8) { da = &s.nx[0].cell(pnx(-1, lane), at.rl); na = 272; }
        else if (lane < 16) { da = &s.ex[0].cell(lane - 8, at.rl); na = 16; }
        else if (at.rl == 0) { da = &s.ny[0].cell(pny(lane - 16, -1), 0); na = 288; }
        else { da = s.ey[0] + lane - 16; na = 16; }
        da[0] = in.h; da[na] = in.e; da[2 * na] = in.n; da[3 * na] = in.t;
    }
    __syncthreads();
    // ---- faces
    auto face = [&](const auto& f) {
        using F = std::remove_cv_t<decltype(f.hi)>;
        const F g = cst<F>(p.g), ga = cst<F>(p.g * (T)0.5), epsi = cst<F>(p.epsi), ef = cst<F>(p.epsface);
        if constexpr (SPLIT) return face_q_split<F, ENGINE>(f, cst<F>(D), g, ga, epsi, ef);
        else return face_q<F, ENGINE>(f, g, ga, epsi, ef);
    };
    V ax;
    // (source-term beds: engine 1 the bed, engine 2 the surface less the depth)
    V zri;
    if constexpr (ENGINE == 1) zri = zb;
    else zri = sub(c[VZS], c[VH]);
    {
        const int on = pnx(x - 1, r);
        FaceQ<V> f;
        f.hI = X.h; f.eI = X.e; f.nI = X.n; f.tI = X.t;
        f.hN = s.nx[0].get(on, l); f.eN = s.nx[1].get(on, l); f.nN = s.nx[2].get(on, l); f.tN = s.nx[3].get(on, l);
        f.hi = f.hsi = c[VH];
        f.hn = f.hsn = s.t[VH].get(o - 1, l);
        f.zri = zri;
        if constexpr (ENGINE == 1) f.zrn = s.zb.get(pz(x - 1, r), l);
        else f.zrn = sub(s.t[VZS].get(o - 1, l), f.hn);
        if constexpr (SUB) {
            if (x == 0 && subf->on[0]) {
                f.hsn = lanes_of<V>(subf->h[0][r], subf->h[0][r + 8], l);
                f.zrn = lanes_of<V>(subf->z[0][r], subf->z[0][r + 8], l);
            }
        }
        const FluxQ<V> q = face(f);
        const int of = pfx(x, r);
        s.fx[0].put(of, l, q.Fh);
        s.fx[1].put(of, l, q.S);
        s.fx[2].put(of, l, q.Ft);
        if (allfaces) s.fxq().put(of, l, q.Fq);
        own.xh = q.Fh; own.xq = q.Fq; own.xt = q.Ft;
        ax = q.a;
    }
    V amax = cst<V>((T)0);
    {
        const int on = pny(x, r - 1);
        FaceQ<V> f;
        f.hI = Y.h; f.eI = Y.e; f.nI = Y.n; f.tI = Y.t;
        f.hN = s.ny[0].get(on, l); f.eN = s.ny[1].get(on, l); f.nN = s.ny[2].get(on, l); f.tN = s.ny[3].get(on, l);
        f.hi = f.hsi = c[VH];
        f.hn = f.hsn = s.t[VH].get(o - 20, l);
        f.zri = zri;
        if constexpr (ENGINE == 1) f.zrn = s.zb.get(pz(x, r - 1), l);
        else f.zrn = sub(s.t[VZS].get(o - 20, l), f.hn);
        if constexpr (SUB) {
            if (r == 0 && l == 0 && subf->on[2]) {  // the bottom face (lane 0 of pair row 0)
                if constexpr (LANES == 1) {
                    f.hsn = subf->h[2][x];
                    f.zrn = subf->z[2][x];
                } else {
                    f.hsn.a = subf->h[2][x];
                    f.zrn.a = subf->z[2][x];
                }
            }
        }
        const FluxQ<V> q = face(f);
        const int of = pfy(x, r);
        s.fy[0].put(of, l, q.Fh);
        s.fy[1].put(of, l, q.S);
        s.fy[2].put(of, l, q.Ft);
        if (allfaces) s.fyq().put(of, l, q.Fq);
        if (r == 0 && (LANES == 2 || l == 1)) {  // face 8, the upper one of row 7
            const int o8 = pfy(x, 8);
            s.fy[0].cell(o8, 0) = lane_of(q.Fh, 1);
            s.fy[1].cell(o8, 0) = lane_of(q.S, 1);
            s.fy[2].cell(o8, 0) = lane_of(q.Ft, 1);
        }
        own.yh = q.Fh; own.yq = q.Fq; own.yt = q.Ft;
        // a cell's dt: the X sweep's and the Y sweep's smaller one, none where the Y face is dry
        if constexpr (SPEED) amax = sel(q.wet, vmax(ax, q.a), cst<V>((T)0));
    }
    // the faces on the right column (pairs of rows) and the top row (pairs of columns)
    // (one face a lane: with a pair in each of half the lanes the other warps wait longer,
    // 428 instead of 408 us per step for 12,288 blocks of the exact build, fast build
    // 740 instead of 729 us for 65,536 blocks, 25.0 instead of 23.9 us in split precision
    // for 1,536; face_q has the same roundings in both forms)
    if (at.extra) {
        const bool isx = (lane & 15) < 8;
        const int q = lane & 7, el = lane >> 4;  // (which of the two cells)
        // the two cells: rows q and q + 8 of the column 16, or row 16 of the columns 2q, 2q + 1
        const int i0 = isx ? pt(BW, q) : pt(2 * q, 8), z0 = isx ? pz(BW, q) : pz(2 * q, 8);
        const int n0 = isx ? pnx(BW - 1, q) : pny(2 * q, 7), nst = isx ? 272 : 288;
        const T *nn = isx ? s.nx[0].a : s.ny[0].a, *ei = isx ? s.ex[0].a : s.ey[0];
        const int d = (isx ? 1 : 20) * LANES, dz = (isx ? 1 : 18) * LANES;
        // element of the cell in an array of n pairs
        auto first = [&](int pr, int n) {
            if constexpr (LANES == 2) return 2 * pr + (isx ? el : 1 + 2 * el);
            else return isx ? pr + el * n : pr + el + n;
        };
        const int ti_ = first(i0, 240), zi_ = first(z0, 180), ni = first(n0, nst / 2);
        const int ii = LANES == 1 && isx ? q + 8 * el : 2 * q + el;
        auto low = [&](int v) { return ei[16 * v + ii]; };
        FaceQ<T> f;
        f.hI = low(0); f.eI = low(1); f.nI = low(2); f.tI = low(3);
        f.hN = nn[ni]; f.eN = nn[ni + nst]; f.nN = nn[ni + 2 * nst]; f.tN = nn[ni + 3 * nst];
        f.hi = f.hsi = s.t[VH].a[ti_];
        f.hn = f.hsn = s.t[VH].a[ti_ - d];
        if constexpr (ENGINE == 1) {
            f.zri = s.zb.a[zi_];
            f.zrn = s.zb.a[zi_ - dz];
        } else {
            f.zri = sub(s.t[VZS].a[ti_], f.hi);
            f.zrn = sub(s.t[VZS].a[ti_ - d], f.hn);
        }
        if constexpr (SUB) {
            const int sd = isx ? 1 : 3;
            const int j0 = isx ? q : 2 * q, j1 = isx ? q + 8 : 2 * q + 1;
            if (subf->on[sd]) {
                f.hsi = lanes_of<T>(subf->h[sd][j0], subf->h[sd][j1], el);
                f.zri = lanes_of<T>(subf->z[sd][j0], subf->z[sd][j1], el);
            }
        }
        const FluxQ<T> w = face(f);
        T *o0 = isx ? s.fx[0].a : s.fy[0].a, *oq = isx ? s.fxq().a : s.fyq().a;
        const int fo = first(isx ? pfx(BW, q) : pfy(2 * q, 8), nst / 2), fq = first(isx ? pfx(BW, q) : pfy(2 * q, 8), 240);
        o0[fo] = w.Fh;
        o0[fo + nst] = w.S;
        o0[fo + 2 * nst] = w.Ft;
        if (allfaces) oq[fq] = w.Fq;
    }
    if constexpr (LANES == 1) return amax;
    else return amax.a > amax.b ? amax.a : amax.b;
}

// The own cells' face values again from shared memory (after boundary segments changed them).
template <class T, int LANES, class V>
__device__ __forceinline__ void reload_faces(SmemQ<T, LANES>& s, const Place<T, LANES>& at, OwnFlux<V>& own)
{
    const int ox = pfx(at.x, at.r), oy = pfy(at.x, at.r);
    own.xh = s.fx[0].get(ox, at.l); own.xq = s.fxq().get(ox, at.l); own.xt = s.fx[2].get(ox, at.l);
    own.yh = s.fy[0].get(oy, at.l); own.yq = s.fyq().get(oy, at.l); own.yt = s.fy[2].get(oy, at.l);
}

// updateEVCPU (src/Advection.cu:160-254), Cartesian, for the own cells.
template <class T, int LANES, class V>
__device__ __forceinline__ void divergence_q(const SmemQ<T, LANES>& s, const StepParams<T>& p, T cmdinv,
                                             const Place<T, LANES>& at, const OwnFlux<V>& own, V hi, V uui, V vvi, V& dh,
                                             V& dhu, V& dhv)
{
    const int fr = pfx(at.x + 1, at.r), ft = pfy(at.x, at.r + 1);
    const V Fhu_r = s.fx[0].get(fr, at.l), Su_r = s.fx[1].get(fr, at.l), Fqvx_r = s.fx[2].get(fr, at.l);
    const V Fhv_t = s.fy[0].get(ft, at.l), Sv_t = s.fy[1].get(ft, at.l), Fquy_t = s.fy[2].get(ft, at.l);
    const V cm = cst<V>(cmdinv), fc = cst<V>(p.fc), nfc = cst<V>(-p.fc);
    dh = mul(mul(cst<V>((T)-1.0), sub(add(sub(Fhu_r, own.xh), Fhv_t), own.yh)), cm);
    // (the Coriolis products fused into the sums; -fc h u is -(fc h u) exactly)
    dhu = mad(sub(sub(add(own.xq, own.yt), Su_r), Fquy_t), cm, mul(mul(fc, hi), vvi));
    dhv = mad(sub(sub(add(own.yq, own.xt), Sv_t), Fqvx_r), cm, mul(mul(nfc, hi), uui));
}

// bndFluxGPUSideCPU (src/Boundary.cu:587-745); state n: the depth in the tile's h, the
// velocities U and W of the model.
template <class T, bool SPLIT, int LANES>
__device__ __forceinline__ void boundaries_q(SmemQ<T, LANES>& s, const DevModel<T>& m, const StepParams<T>& p, int ib,
                                             double tbnd, int tid, const T* U, const T* W, T D = (T)0)
{
    if (tid >= 64) return;
    const int side = tid >> 4, t = tid & 15;
    const int k = m.bndseg[ib * 4 + side];
    if (k < 0) return;
    const SegDev sg = m.segs[k];
    if (sg.type == 1) return;
    double zsbnd = 0.0;
    if (!isnan(p.zsinit)) zsbnd = p.zsinit;
    T taper = (T)1.0;
    if (sg.n > 0) {
        if (p.bndtaper > 0.0) taper = (T)fmin((tbnd - p.inittime) / p.bndtaper, 1.0);
        zsbnd = series_at(m.seg_t + sg.off, m.seg_wl + sg.off, sg.n, tbnd, sg.sorted != 0);
    }
    const int isright = side == 0 ? -1 : side == 1 ? 1 : 0;
    const int istop = side == 2 ? 1 : side == 3 ? -1 : 0;
    int ix, iy, inx, iny;
    if (isright == 0) { ix = t; iy = istop < 0 ? 0 : BW; }
    else { iy = t; ix = isright < 0 ? 0 : BW; }
    if (isright < 0) { inx = ix + 1; iny = iy; }
    else if (isright > 0) { inx = ix - 1; iny = iy; }
    else if (istop < 0) { inx = ix; iny = iy + 1; }
    else { inx = ix; iny = iy - 1; }
    const T sign = (T)isright + (T)istop;
    float zsb = (float)zsbnd;
    zsb = (float)((double)zsb + p.zsoffset);
    const T H0 = BGF_ROW(s.t[VH], pt, ix, iy), H1 = BGF_ROW(s.t[VH], pt, inx, iny);
    // (split precision: beds zb + D and depths D + h'; zs is the surface either way)
    const T zsi = BGF_ROW(s.zb, pz, ix, iy) + H0;
    const T zsinside = BGF_ROW(s.zb, pz, inx, iny) + H1;
    const T hinside = SPLIT ? D + H1 : H1;
    const T uninside = (isright != 0 ? U : W)[(size_t)ib * 256 + iny * 16 + inx];
    const T hface = SPLIT ? D + H0 : H0;
    const T zsX = (T)(((double)((T)zsb + (T)0.0) - 0.5 * (double)(zsi + zsinside)) * (double)taper +
                      0.5 * (double)(zsi + zsinside));
    float* qm = m.qmean + ib * 64 + side * 16 + t;
    T qmean = (T)*qm;
    // the face itself (mass flux, and the momentum flux of its inner side) and the one a cell
    // further in (the source side of the other direction)
    T *pF, *pG, *pS;
    if (isright != 0) {
        pF = &BGF_ROW(s.fx[0], pfx, ix, iy);
        pG = isright < 0 ? &BGF_ROW(s.fxq(), pfx, ix, iy) : &BGF_ROW(s.fx[1], pfx, ix, iy);
        pS = isright < 0 ? &BGF_ROW(s.fx[1], pfx, inx, iny) : &BGF_ROW(s.fxq(), pfx, inx, iny);
    } else {
        pF = &BGF_ROW(s.fy[0], pfy, ix, iy);
        pG = istop < 0 ? &BGF_ROW(s.fyq(), pfy, ix, iy) : &BGF_ROW(s.fy[1], pfy, ix, iy);
        pS = istop < 0 ? &BGF_ROW(s.fy[1], pfy, inx, iny) : &BGF_ROW(s.fyq(), pfy, inx, iny);
    }
    T F = *pF, S = *pS;
    const T G = *pG;
    const T factime = M<T>::fmin_((T)(p.dtparam / p.bndfiltertime), (T)1.0);
    const T facrel = (T)1.0 - M<T>::fmin_((T)(p.dtparam / p.bndrelaxtime), (T)1.0);
    if (sg.type == 0) {
        F = (T)0.0;
        S = G;
    } else if (sg.type == 3) {
        if ((double)hface > p.eps_d || zsX > zsi) {
            abs1dq<T>(p.g, sign, factime, facrel, zsi, zsX, hface, qmean, F);
        } else {
            F = (T)0.0; S = G; qmean = (T)0.0;
        }
        *qm = (float)qmean;
    } else if (sg.type == 2) {
        if ((double)hface > p.eps_d || zsX > zsi) {
            dirichlet1q<T>(p.g, sign, zsX, zsinside, hinside, uninside, F);
        } else {
            F = (T)0.0; S = G; qmean = (T)0.0;
        }
        *qm = (float)qmean;
    }
    *pF = F;
    *pS = S;
}

// The block's dt from the largest wave speed of its cells into the scenario's minimum.  A
// cell whose state is not finite counts as an infinite speed (dt 0 ends the scenario).
template <class T> __device__ __forceinline__ T finite_speed(T h, T u, T v, T a)
{
    return isfinite(h) && isfinite(u) && isfinite(v) ? a : (T)INFINITY;
}
template <class T> __device__ __forceinline__ T finite_speed(V2<T> h, V2<T> u, V2<T> v, T a)
{
#if BGF_FAST
    if constexpr (sizeof(T) == 4) {
        // one test per cell: the sum is finite exactly when h, u and v are (a NaN or an
        // infinity carries through it; finite states are far below the float range)
        const V2<T> q = add(add(h, u), v);
        return isfinite(q.a) && isfinite(q.b) ? a : (T)INFINITY;
    }
#endif
    return finite_speed<T>(h.a, u.a, v.a, finite_speed<T>(h.b, u.b, v.b, a));
}
template <class T, int LANES> __device__ __forceinline__ void warp_max(SmemQ<T, LANES>& s, int tid, T a)
{
    for (int o = 16; o > 0; o >>= 1) {
        const T q = __shfl_xor_sync(0xffffffffu, a, o);
        a = q > a ? q : a;
    }
    if ((tid & 31) == 0) s.red[tid >> 5] = a;
}
template <class T, int LANES>
__device__ __forceinline__ void block_dt(const SmemQ<T, LANES>& s, const StepParams<T>& p, T delta, unsigned long long* slot)
{
    T a = s.red[0];
    for (int k = 1; k < Quad<T, LANES>::NW; k++) a = s.red[k] > a ? s.red[k] : a;
    const T cd = p.CFL * delta;
    atomicMin(slot, dt_bits(a > (T)0 ? dv(cd, a) : inv_epsi<T>()));
}

// add_rivers out of line: few scenarios have rivers, and the inlined copies crowd the
// corrector's instruction cache.
template <class T>
__device__ __noinline__ T river_cell(const RiverDev* rivers, const double* riv_t, const double* riv_q, int first, int nriver,
                                     T levdx, double xo, double yo, int x, int y, T dh, double time)
{
    return add_rivers_cell<T>(rivers, riv_t, riv_q, first, nriver, levdx, xo, yo, x, y, dh, time);
}
template <class T>
__device__ __forceinline__ T add_rivers_q(const DevModel<T>& m, const StepParams<T>& p, int ib, int x, int y, T dh, double time)
{
    return river_cell<T>(m.rivers, m.riv_t, m.riv_q, p.riv_first, p.nriver, calcres<T>(p.delta0, m.level[ib]),
                         p.xo_d + m.bxo[ib], p.yo_d + m.byo[ib], x, y, dh, time);
}

// The full step and the friction of one cell as the multi-level chain's other kernels
// (StageState) make them: plain divisions and cube root.
template <class T>
__device__ __forceinline__ void plain_step(const StepParams<T>& p, T dt, T cf, T hold, T uold, T vold, T dh, T dhu, T dhv,
                                           T& ho, T& uo, T& vo)
{
    advance<T>(dt, p.eps, p.eps_d, p.forcemass != 0, hold, uold, vold, dh, dhu, dhv, ho, uo, vo);
    bottom_friction<T>(p.frictionmodel, p.g, p.eps, dt, cf, ho, uo, vo);
}

// Full step of the own cells from state n (AdvkernelCPU with evolv), then friction on the
// result and rain; the next state goes to buffer nxt.  PLAIN: with the compiler's divisions
// (fast build: full range) instead of products with the reciprocal, cell by cell.
template <class T, bool SPLIT, int LANES, bool PLAIN = false, class V>
__device__ __forceinline__ void full_step(const DevModel<T>& m, const StepParams<T>& p, int ib, const Place<T, LANES>& at,
                                          size_t g, int nxt, T dt, T delta, T D, T rainv, double time, V hold, V uold,
                                          V vold, V dh, V dhu, V dhv)
{
    const bool fm = p.forcemass != 0;
    const V Dv = cst<V>(D);
    const V cfv = p.has_cf ? own_of<V>(m.cf, g, 128, at.l) : cst<V>(p.cf);
    V ho, uo, vo;
    if constexpr (PLAIN && LANES == 1) {
        plain_step<T>(p, dt, cfv, hold, uold, vold, dh, dhu, dhv, ho, uo, vo);
    } else if constexpr (PLAIN) {
        plain_step<T>(p, dt, cfv.a, hold.a, uold.a, vold.a, dh.a, dhu.a, dhv.a, ho.a, uo.a, vo.a);
        plain_step<T>(p, dt, cfv.b, hold.b, uold.b, vold.b, dh.b, dhu.b, dhv.b, ho.b, uo.b, vo.b);
    } else {
        if constexpr (SPLIT) advance_split_v<V>(dt, p.eps, fm, Dv, hold, uold, vold, dh, dhu, dhv, ho, uo, vo);
        else advance_v<V>(dt, p.eps, p.eps_d, fm, hold, uold, vold, dh, dhu, dhv, ho, uo, vo);
        // (split precision: friction on the full depth; the deviation is not changed by it)
        friction_v<V>(p.frictionmodel, p.g, p.eps, dt, cfv, SPLIT ? add(Dv, ho) : ho, uo, vo);
    }
    auto quot = [](V x, V y) {
        if constexpr (!PLAIN) return dv(x, y);
        else if constexpr (LANES == 1) return x / y;
        else return V{x.a / y.a, x.b / y.b};
    };
    if (p.has_rain) {
        // AddrainforcingImplicitCPU (src/Updateforcing.cu:530-580): the rain rate at
        // the start of the step, uniform or gridded
        V Rainhh;
        const V mask = m.rainmask ? own_of<V>(m.rainmask, g, 128, at.l) : cst<V>((T)1);
        if (p.rain_map) {
            const T xc = (T)p.xo_d + (T)m.bxo[ib] + (T)at.x * delta;
            auto rate = [&](int y) {
                return rain_map_at<T>(m.rmap, xc, (T)p.yo_d + (T)m.byo[ib] + (T)y * delta, time);
            };
            if constexpr (LANES == 1) Rainhh = rate(at.r + 8 * at.l);
            else Rainhh = V{rate(at.r), rate(at.r + 8)};
            const V rr = quot(quot(Rainhh, cst<V>((T)1000.0)), cst<V>((T)3600.0));
            Rainhh = mul(vmax(mul(rr, cst<V>(dt)), cst<V>((T)0.0)), mask);
        } else {
            Rainhh = mul(cst<V>(rainv), mask);  // (the block's uniform depth, above)
        }
        const V hi = SPLIT ? add(Dv, ho) : ho;
        const V qvol = quot(hi, add(hi, Rainhh));
        ho = add(ho, Rainhh);
        typename LaneOf<V>::Mask wet;
        if constexpr (LANES == 1) wet = (double)hi > p.eps_d;
        else wet = M2{(double)hi.a > p.eps_d, (double)hi.b > p.eps_d};
        uo = sel(wet, mul(uo, qvol), uo);
        vo = sel(wet, mul(vo, qvol), vo);
    }
    put_own(m.h[nxt], g, at.l, ho);
    put_own(m.u[nxt], g, at.l, uo);
    put_own(m.v[nxt], g, at.l, vo);
    if (m.hmax) {
        const V hf = SPLIT ? add(Dv, ho) : ho;  // the full depth
        const V hx = own_of<V>(m.hmax, g, 128, at.l);
        put_own(m.hmax, g, at.l, sel(gt(hf, hx), hf, hx));
    }
}

// Programmatic dependent launch: a step kernel lets the next one start as soon as its own
// last blocks have, and waits, after the loads that no kernel of a run changes, until the
// one before it has completed (every block waits, so completion is transitive along the
// chain).  Both do nothing in a launch without the
// attribute.  The trigger comes late, after the faces: next blocks that start while a
// kernel is still spread thinly over the SMs would share them unevenly (425 blocks of
// the exact build: 36 us per step with the trigger first, 31 us without, 31 us so).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------- kernels

// Predictor of block w by the CTA's threads (the caller puts a barrier between two blocks).
template <class T, int ENGINE, bool POOL, bool SPLIT, int LANES>
__device__ __forceinline__ void flux_block(SmemQ<T, LANES>& s, const DevModel<T>& m, const StepParams<T>& p0, int parity, int w,
                                           int tid)
{
    using V = typename ValOf<T, LANES>::V;
    const Place<T, LANES> at(tid, w);
    const int ib = m.regular_nbx > 0 ? w : m.active[w];
    // the bed, the bed gradients and the ring cell's source do not depend on the time slot:
    // their loads are in flight while it arrives
    const T* zbt = m.zb + (size_t)ib * 324;
    V zb = own_of<V>(zbt, hi18(at.x, at.r), 8 * 18, at.l);
    BedGradQ<T, LANES> bg;
    load_bedgrad_q<T, ENGINE, LANES>(m, ib, at, bg);
    int rx, ry, rb, sx, sy;
    ring_cell<T>(m, ib, tid & 127, rx, ry, rb, sx, sy);
    const size_t gr = (size_t)rb * 256 + sy * 16 + sx;
    const bool ring2 = rx < -1 || rx > BW || ry < -1 || ry > BW;
    const T rz = ring2 ? m.zb[(size_t)rb * 324 + hi18(sx, sy)] : zbt[hi18(rx, ry)];
    const int sc = POOL ? m.scen[ib] : 0;
    const StepParams<T>& p = params_ref<POOL>(m, p0, sc);
    const T delta = calcres<T>(p.delta0, m.level[ib]);
    const T D = SPLIT ? m.datum[ib] : (T)0;  // split precision: the block's datum
    const bool segs = block_has_segments<T>(m, ib);
    pdl_wait();
    const TimeState ts = m.time[2 * sc + parity];
    if (!step_live(ts)) return;
    const T* H = m.h[ts.cur];
    const T* U = m.u[ts.cur];
    const T* W = m.v[ts.cur];
    const size_t g = (size_t)ib * 256 + at.r * 16 + at.x;
    V c[4];
    c[VH] = own_of<V>(H, g, 128, at.l);
    c[VU] = own_of<V>(U, g, 128, at.l);
    c[VV] = own_of<V>(W, g, 128, at.l);
    if (LANES == 2 || tid < 128) {
        T hv = H[gr];
        const T uv = U[gr], vv = W[gr];
        // split precision: a neighbour's deviation in this block's datum (datums are
        // whole metres, so the difference is exact)
        if (SPLIT && rb != ib) hv = hv + (m.datum[rb] - D);
        store_ring<T, LANES>(s, rx, ry, hv, uv, vv, SPLIT ? rz + D : rz);
    }
    if (SPLIT) zb = add(zb, cst<V>(D));
    c[VZS] = add(zb, c[VH]);
    store_own<T, LANES>(s, at, c, zb);
    __syncthreads();
    OwnFlux<V> own;
    T a = tile_faces<T, ENGINE, LANES, SPLIT, true, false>(s, p, delta, at, c, zb, bg, segs, own, D);
    a = finite_speed(c[VH], c[VU], c[VV], a);
    warp_max<T, LANES>(s, tid, a);
    pdl_trigger();
    __syncthreads();
    // boundary segments (FlowbndFlux) after the dt, at t + dt_prev / 2 as FlowCPU does
    if (segs) {
        boundaries_q<T, SPLIT, LANES>(s, m, p, ib, ts.totaltime + ts.dt * 0.5, tid, U, W, D);
        __syncthreads();
        reload_faces<T, LANES>(s, at, own);
    }
    if (tid == 0) block_dt<T, LANES>(s, p, delta, &m.dtmin[2 * sc + parity]);
    V dh, dhu, dhv;
    divergence_q<T, LANES>(s, p, (T)1.0 / ((T)1.0 * delta), at, own, SPLIT ? add(cst<V>(D), c[VH]) : c[VH], c[VU], c[VV], dh,
                           dhu, dhv);
    put_own(m.dh, g, at.l, dh);
    put_own(m.dhu, g, at.l, dhu);
    put_own(m.dhv, g, at.l, dhv);
}

// Corrector of block w by the CTA's threads (the caller puts a barrier between two blocks).
template <class T, int ENGINE, bool POOL, bool SPLIT, int LANES>
__device__ __forceinline__ void update_block(SmemQ<T, LANES>& s, const DevModel<T>& m, const StepParams<T>& p0, int parity,
                                             int w, int tid)
{
    using V = typename ValOf<T, LANES>::V;
    const Place<T, LANES> at(tid, w);
    const int ib = m.regular_nbx > 0 ? w : m.active[w];
    // the bed and the ring cell's source depend on no kernel of the run, the predictor's
    // tendencies not on the time slot (only the state buffer does): their loads are in
    // flight while it arrives
    const T* zbt = m.zb + (size_t)ib * 324;
    const size_t g = (size_t)ib * 256 + at.r * 16 + at.x;
    V zb = own_of<V>(zbt, hi18(at.x, at.r), 8 * 18, at.l);
    BedGradQ<T, LANES> bg;
    load_bedgrad_q<T, ENGINE, LANES>(m, ib, at, bg);
    int rx, ry, rb, sx, sy;
    ring_cell<T>(m, ib, tid & 127, rx, ry, rb, sx, sy);
    const size_t gr = (size_t)rb * 256 + sy * 16 + sx;
    const bool ring2 = rx < -1 || rx > BW || ry < -1 || ry > BW;
    const T rz = ring2 ? m.zb[(size_t)rb * 324 + hi18(sx, sy)] : zbt[hi18(rx, ry)];
    const int sc = POOL ? m.scen[ib] : 0;
    const StepParams<T>& p = params_ref<POOL>(m, p0, sc);
    const T delta = calcres<T>(p.delta0, m.level[ib]);
    const T D = SPLIT ? m.datum[ib] : (T)0;  // split precision: the block's datum
    const V Dv = cst<V>(D);
    const bool segs = block_has_segments<T>(m, ib);
    const bool lead = POOL ? m.lead[ib] != 0 : w == 0;
    pdl_wait();
    V ddh = own_of<V>(m.dh, g, 128, at.l);
    const V ddhu = own_of<V>(m.dhu, g, 128, at.l), ddhv = own_of<V>(m.dhv, g, 128, at.l);
    T rdh = m.dh[gr];
    const T rdhu = m.dhu[gr], rdhv = m.dhv[gr];
    // the predictor's dt minimum (read by thread 0) does not depend on it either
    const unsigned long long dtbits = tid == 0 ? m.dtmin[2 * sc + parity] : 0ull;
    const TimeState ts = m.time[2 * sc + parity];
    if (!step_live(ts)) {
        if (lead && tid == 0) {
            TimeState nt = ts;
            nt.done = 1;
            m.time[2 * sc + (parity ^ 1)] = nt;
        }
        return;
    }
    if (tid == 0) {
        const T dt0 = step_dt<T>(ts, dtbits);
        s.dtv = dt0;
        if (p.has_rain && !p.rain_map) {
            // uniform rain (AddrainforcingImplicitCPU, src/Updateforcing.cu:530-580): the
            // rate at the start of the step and its depth over the step, the same for
            // every cell of the scenario, once per block instead of once per thread
            const T r = (T)series_at(m.rain_t + p.rain_off, m.rain_r + p.rain_off, p.rain_n, ts.totaltime,
                                     p.rain_sorted != 0);
            s.rainv = M<T>::fmax_(dv(dv(r, (T)1000.0), (T)3600.0) * dt0, (T)0.0);
        }
    }
    const T* H = m.h[ts.cur];
    const T* U = m.u[ts.cur];
    const T* W = m.v[ts.cur];
    const V hold = own_of<V>(H, g, 128, at.l), uold = own_of<V>(U, g, 128, at.l), vold = own_of<V>(W, g, 128, at.l);
    const T rh = H[gr], ru = U[gr], rv = W[gr];
    __syncthreads();  // s.dtv
    const T dt = s.dtv;
    const double dtd = (double)dt;
    const T halfdt = dt * (T)0.5;
    const bool fm = p.forcemass != 0;
    // rivers: the predictor's source of a cell (AddRiverForcing after updateEV)
    auto rivers = [&](V d) {
        if constexpr (LANES == 1) return add_rivers_q<T>(m, p, ib, at.x, at.r + 8 * at.l, d, ts.totaltime);
        else return V{add_rivers_q<T>(m, p, ib, at.x, at.r, d.a, ts.totaltime),
                      add_rivers_q<T>(m, p, ib, at.x, at.r + 8, d.b, ts.totaltime)};
    };
    if (p.nriver > 0) {
        ddh = rivers(ddh);
        rdh = add_rivers_q<T>(m, p, rb, sx, sy, rdh, ts.totaltime);
    }
    V c[4];
    if constexpr (SPLIT) {
        advance_split_v<V>(halfdt, p.eps, fm, Dv, hold, uold, vold, ddh, ddhu, ddhv, c[VH], c[VU], c[VV]);
        zb = add(zb, Dv);
    } else {
        advance_v<V>(halfdt, p.eps, p.eps_d, fm, hold, uold, vold, ddh, ddhu, ddhv, c[VH], c[VU], c[VV]);
    }
    c[VZS] = add(zb, c[VH]);
    store_own<T, LANES>(s, at, c, zb);
    if (LANES == 2 || tid < 128) {
        T ho, uo, vo;
        if constexpr (SPLIT) {
            // the source cell's half step in its own datum, then in this block's
            const T Ds = rb == ib ? D : m.datum[rb];
            advance_split<T>(halfdt, p.eps, fm, Ds, rh, ru, rv, rdh, rdhu, rdhv, ho, uo, vo);
            if (rb != ib) ho = ho + (Ds - D);
        } else {
            advance_v<T>(halfdt, p.eps, p.eps_d, fm, rh, ru, rv, rdh, rdhu, rdhv, ho, uo, vo);
        }
        store_ring<T, LANES>(s, rx, ry, ho, uo, vo, SPLIT ? rz + D : rz);
    }
    __syncthreads();
    OwnFlux<V> own;
    (void)tile_faces<T, ENGINE, LANES, SPLIT, false, false>(s, p, delta, at, c, zb, bg, segs, own, D);
    pdl_trigger();
    __syncthreads();
    if (segs) {  // interior blocks skip the step and its barriers
        // the segments read state n: its depth takes the half-step depth's place in the tile
        s.t[VH].put(pt(at.x, at.r), at.l, hold);
        if (LANES == 2 || tid < 128) {
            // (the ring cell's place once more: held over the faces it would cost registers)
            ring_cell<T>(m, ib, tid & 127, rx, ry, rb, sx, sy);
            T hv = H[(size_t)rb * 256 + sy * 16 + sx];
            if (SPLIT && rb != ib) hv = hv + (m.datum[rb] - D);
            BGF_ROW(s.t[VH], pt, rx, ry) = hv;
        }
        __syncthreads();
        boundaries_q<T, SPLIT, LANES>(s, m, p, ib, ts.totaltime + dtd, tid, U, W, D);
        __syncthreads();
        reload_faces<T, LANES>(s, at, own);
    }
    V dh, dhu, dhv;
    divergence_q<T, LANES>(s, p, (T)1.0 / ((T)1.0 * delta), at, own, SPLIT ? add(Dv, c[VH]) : c[VH], c[VU], c[VV], dh, dhu,
                           dhv);
    if (p.nriver > 0) dh = rivers(dh);
    const int nxt = ts.cur ^ 1;
    full_step<T, SPLIT, LANES>(m, p, ib, at, g, nxt, dt, delta, D, s.rainv, ts.totaltime, hold, uold, vold, dh, dhu, dhv);
    if (lead && tid == 0)
        m.time[2 * sc + (parity ^ 1)] = next_time_state<T>(ts, p, dtd, nxt, m.dtmin + 2 * sc, parity);
}

template <class T, int ENGINE, bool POOL, bool SPLIT, int LANES>
__global__ void __launch_bounds__(Quad<T, LANES>::NT, Quad<T, LANES>::ctas)
    fluxq_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ StepParams<T> p0, int parity)
{
    extern __shared__ __align__(16) unsigned char smem_rawq[];
    for (int w = blockIdx.x; w < m.nblk; w += gridDim.x) {
        flux_block<T, ENGINE, POOL, SPLIT, LANES>(*reinterpret_cast<SmemQ<T, LANES>*>(smem_rawq), m, p0, parity, w, threadIdx.x);
        if (w + (int)gridDim.x < m.nblk) __syncthreads();  // the tile is reused by the next block
    }
}

template <class T, int ENGINE, bool POOL, bool SPLIT, int LANES>
__global__ void __launch_bounds__(Quad<T, LANES>::NT, Quad<T, LANES>::ctas)
    updateq_kernel(const __grid_constant__ DevModel<T> m, const __grid_constant__ StepParams<T> p0, int parity)
{
    extern __shared__ __align__(16) unsigned char smem_rawq[];
    for (int w = blockIdx.x; w < m.nblk; w += gridDim.x) {
        update_block<T, ENGINE, POOL, SPLIT, LANES>(*reinterpret_cast<SmemQ<T, LANES>*>(smem_rawq), m, p0, parity, w,
                                                    threadIdx.x);
        if (w + (int)gridDim.x < m.nblk) __syncthreads();  // the tile is reused by the next block
    }
}
