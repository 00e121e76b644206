// mgp_sweep.cuh -- Gauss-Seidel sweeps of a window of a level by one CTA: the
// device routines of mgp_sweep.cu's kernels, which the coarse cycle
// (mgp_kernels.cu) also runs on the levels it holds.
#pragma once

#include "mgp_kernels.cuh"

namespace mgp {

namespace {

// A CTA's shape: NI warps own the window's blocks, a thread a block, LB blocks (2
// LB columns) a row (threads past the last whole row have none); with kSep four
// more warps serve the domain's sides.
template <class T_, int NI_, int LB_, bool kSep_, int kMinBlocks_>
struct Shape {
    using T = T_;
    static constexpr int NI = NI_, LB = LB_, kMinBlocks = kMinBlocks_;
    static constexpr bool kSep = kSep_;
    static constexpr int NR = 32 * NI / LB;                  // block rows
    static constexpr int kThreads = 32 * (NI + (kSep ? 4 : 0));
    static constexpr int WX = 2 * LB, WY = 2 * NR;           // window
    static constexpr int P = LB + 2;                         // blocks per plane row, one spare either side
    static constexpr int PS = P * (NR + 2);                  // one plane
    static_assert(WX <= 64 && WY <= 64 && NI >= 4, "a warp holds a side, two cells a lane");
    // largest tile for K sweeps a launch
    static constexpr int tx(int k) { return WX - (8 * k + 2); }
    static constexpr int ty(int k) { return WY - (8 * k + 4); }
};

// Programmatic dependent launch: a grid launched with the programmatic
// serialization attribute may start before the grid ahead of it in the stream
// has finished; griddepcontrol.wait returns once that grid has completed and
// its writes are visible (at once when there is none), and launch_dependents
// lets the next such grid start as SM resources free up.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Barrier of the four warps that serve the sides, and of the whole CTA (the
// two roles reach it at different places in the code).
__device__ __forceinline__ void boundary_sync() {
    __syncwarp();
    asm volatile("bar.sync 1, 128;" ::: "memory");
}
__device__ __forceinline__ void cta_sync() {
    __syncwarp();
    asm volatile("bar.sync 0;" ::: "memory");
}

template <class T>
struct Pair;
template <>
struct Pair<float> {
    using type = float2;
};
template <>
struct Pair<double> {
    using type = double2;
};

// Elements p[0] (if a) and p[1] (if b; b implies a).  kVec: p is aligned to a
// pair.  kConst: the memory is not written while the kernel runs or by the
// kernel ahead of it.
template <bool kVec, bool kConst, class T>
__device__ __forceinline__ void load_pair(const T* p, bool a, bool b, T& v0, T& v1) {
    using V = typename Pair<T>::type;
    if (kVec && b) {
        const V v = kConst ? __ldg(reinterpret_cast<const V*>(p)) : *reinterpret_cast<const V*>(p);
        v0 = v.x;
        v1 = v.y;
    } else {
        if (a) v0 = kConst ? __ldg(p) : p[0];
        if (b) v1 = kConst ? __ldg(p + 1) : p[1];
    }
}

// A plane index is the sum of a term of the window column x and one of the row
// y, -1 <= x <= WX, -1 <= y <= WY.
template <class C>
__device__ __forceinline__ int x_term(int x) {
    return (x & 1) * C::PS + (x >> 1);
}
template <class C>
__device__ __forceinline__ int y_term(int y) {
    return (y & 1) * 2 * C::PS + (y >> 1) * C::P + C::P + 1;
}

// The part of the grid a CTA works on.
struct Window {
    int ox, oy, wx1, wy1;      // cells [ox, wx1) x [oy, wy1)
    int X0, X1, Y0, Y1;        // its tile
    bool xl, xh, yl, yh;       // sides of the domain in the window
    __device__ __forceinline__ bool any() const { return xl || xh || yl || yh; }
    // The tile and its halo (cells left, right, below, above), clipped to the grid.
    __device__ __forceinline__ void set(int x0, int x1, int y0, int y1, int l, int r, int d, int u, int nx, int ny) {
        X0 = x0, X1 = x1, Y0 = y0, Y1 = y1;
        ox = max(0, X0 - l), wx1 = min(nx, X1 + r);
        oy = max(0, Y0 - d), wy1 = min(ny, Y1 + u);
        xl = ox == 0, xh = wx1 == nx, yl = oy == 0, yh = wy1 == ny;
    }
};

// phi at the start of a launch's second and later sweeps: the window where it
// holds (i,j), else global memory (a stored ghost; a launch of several sweeps has
// a periodic side only where one window holds the level).
template <class C>
struct StartLoad {
    using T = typename C::T;
    const T* s;
    const Window& w;
    DFT<T> pin;
    __device__ __forceinline__ T operator()(int i, int j) const {
        if (i >= w.ox && i < w.wx1 && j >= w.oy && j < w.wy1) return s[x_term<C>(i - w.ox) + y_term<C>(j - w.oy)];
        return AT(pin, i, j);
    }
};

// What a thread keeps of its 2 x 2 block: x-faces [row][face], y-faces
// [face][column], inverse diagonal, right-hand side and phi [row][column].
// FP64: Jgup_xy and Jgup_yx times 1/4 (the first product lap9f forms, so the
// same bits).  FP32: every face value times its two grid factors (dx^-2, or
// dx^-1 dy^-1 / 4), one rounding, and the inverse diagonal times omega.
template <class T>
struct Block {
    T xx[2][3], xy[2][3], yx[3][2], yy[3][2], d[2][2], f[2][2], p[2][2];
};

// The update of the block's cell (CX, CY), an interior cell; s is the block's
// place in plane 0.
template <class C, int CX, int CY, class T>
__device__ __forceinline__ T update(const Block<T>& k, const T* s, T idx, T idy, T om, T om1) {
    const auto N = [&](int dx, int dy) -> T {   // compile-time dx, dy
        const int x = CX + dx, y = CY + dy;
        if (x >= 0 && x <= 1 && y >= 0 && y <= 1) return k.p[y][x];
        return s[((y & 1) * 2 + (x & 1)) * C::PS + (y >> 1) * C::P + (x >> 1)];
    };
    const T p = k.p[CY][CX], pe = N(1, 0), pw = N(-1, 0), pn = N(0, 1), ps = N(0, -1);
    const T ene = N(1, 1), enw = N(-1, 1), ese = N(1, -1), esw = N(-1, -1);
    if constexpr (sizeof(T) == 8) {   // lap9f's operations in their order (P2:1768-1771 for the update)
        const T xfe = k.xx[CY][CX + 1] * (pe - p) * idx + k.xy[CY][CX + 1] * (ene - ese + pn - ps) * idy;
        const T xfw = k.xx[CY][CX] * (p - pw) * idx + k.xy[CY][CX] * (pn - ps + enw - esw) * idy;
        const T yfn = k.yy[CY + 1][CX] * (pn - p) * idy + k.yx[CY + 1][CX] * (ene - enw + pe - pw) * idx;
        const T yfs = k.yy[CY][CX] * (p - ps) * idy + k.yx[CY][CX] * (pe - pw + ese - esw) * idx;
        const T lphi = (xfe - xfw) * idx + (yfn - yfs) * idy;
        const T newphi = p + (k.f[CY][CX] - lphi) * k.d[CY][CX];
        return om * newphi + om1 * p;
    } else {
        const T ty = pn - ps, tx = pe - pw;
        T x = k.xx[CY][CX + 1] * (pe - p);
        x = __fmaf_rn(k.xx[CY][CX], pw - p, x);
        x = __fmaf_rn(k.xy[CY][CX + 1], (ene - ese) + ty, x);
        x = __fmaf_rn(k.xy[CY][CX], (esw - enw) - ty, x);
        T y = k.yy[CY + 1][CX] * (pn - p);
        y = __fmaf_rn(k.yy[CY][CX], ps - p, y);
        y = __fmaf_rn(k.yx[CY + 1][CX], (ene - enw) + tx, y);
        y = __fmaf_rn(k.yx[CY][CX], (esw - ese) - tx, y);
        return __fmaf_rn((k.f[CY][CX] - x) - y, k.d[CY][CX], p);
    }
}

// ---- the cells along the domain's sides ------------------------------------ //
// A warp serves each side the window holds: its ghosts, its edge cells colour
// by colour and one corner.  A side is described by its tangential direction t
// (x on the y sides, y on the x sides) and its normal n; the cell formulas are
// gather9's and lap9f's with t for x and n for y, which on the x sides are the
// same operations by the symmetry of the operator under exchanging x and y.
// A lane keeps two neighbouring cells of the side, one of each colour, and their
// operator.  These passes are a serial chain of single warps (about 4 cycles an
// instruction), four times the interior's 745 cycles a sweep in FP64, so every
// instruction that does not depend on phi is made once, before the sweeps, and
// the rest are few: places known at compile time, ghosts read before the interior
// colours and written beside them, the FP32 operator folded into nine weights.  A
// sweep of 32^2 cells: 2.6 -> 2.05 us in FP64, 2.0 -> 1.3 in FP32.
//
// The operator at a side's cells comes from their owners through shared
// memory: value q of cell a along side t at [(t * kStrip + q) * kAlong + a].
constexpr int kStrip = 10, kAlong = 64;
enum { Q_TT1, Q_TT0, Q_TN1, Q_TN0, Q_NN1, Q_NN0, Q_NT1, Q_NT0, Q_D, Q_F };   // 1: the high face, 0: the low face
// Weights by cell: plus and minus along the side; the cell itself, one and two inward; the ghost.
enum { W_PP, W_PM, W_P1, W_M1, W_P2, W_M2, W_I1, W_I2, W_GH, W_D, W_F };

template <int CX, int CY, class T>
__device__ __forceinline__ void strip_write(T* q, const Block<T>& k, bool yside) {
    const T xe = k.xx[CY][CX + 1], xw = k.xx[CY][CX], ce = k.xy[CY][CX + 1], cw = k.xy[CY][CX];
    const T yn = k.yy[CY + 1][CX], ys = k.yy[CY][CX], dn = k.yx[CY + 1][CX], ds = k.yx[CY][CX];
    q[Q_TT1 * kAlong] = yside ? xe : yn;
    q[Q_TT0 * kAlong] = yside ? xw : ys;
    q[Q_TN1 * kAlong] = yside ? ce : dn;
    q[Q_TN0 * kAlong] = yside ? cw : ds;
    q[Q_NN1 * kAlong] = yside ? yn : xe;
    q[Q_NN0 * kAlong] = yside ? ys : xw;
    q[Q_NT1 * kAlong] = yside ? dn : ce;
    q[Q_NT0 * kAlong] = yside ? ds : cw;
    q[Q_D * kAlong] = k.d[CY][CX];
    q[Q_F * kAlong] = k.f[CY][CX];
}

// The corner (kHX, kHY) of the domain, its operator in a y side's strip at q; x
// and y: plane terms of the ghosts, the side's cells and the next two inward.
template <bool kHX, bool kHY, class T>
__device__ __forceinline__ void corner_cell(T* S, const T* q, const int* x, const int* y, const GeoT<T>& g,
                                            const BCd& b, int homog, int i, int j, T om, T om1) {
    const T three = T(3.0), half = T(0.5);
    const T p = S[x[1] + y[1]], a = S[x[2] + y[1]], c = S[x[1] + y[2]], ac = S[x[2] + y[2]];   // a, c: x, y inward
    const T gx = S[x[0] + y[1]], gy = S[x[1] + y[0]];
    const T o = three * (p - a) + S[x[3] + y[1]], u = three * (p - c) + S[x[1] + y[3]];   // outward in x, in y
    const T oc = three * (c - ac) + S[x[3] + y[2]], au = three * (a - ac) + S[x[2] + y[3]];
    const T ou = half * ((three * (u - au) + S[x[3] + y[0]]) + (three * (o - oc) + S[x[0] + y[3]]));
    St9T<T> st;
    st.p = p;
    st.pe = kHX ? gx : a;
    st.pw = kHX ? a : gx;
    st.pn = kHY ? gy : c;
    st.ps = kHY ? c : gy;
    st.ee = kHX ? o : a;
    st.ew = kHX ? a : o;
    st.en = kHY ? u : c;
    st.es = kHY ? c : u;
    const T ni = kHY ? au : ac, si = kHY ? ac : au, no = kHY ? ou : oc, so = kHY ? oc : ou;   // x inward, outward
    st.ene = kHX ? no : ni;
    st.enw = kHX ? ni : no;
    st.ese = kHX ? so : si;
    st.esw = kHX ? si : so;
    FacesT<T> fc;
    fc.xxe = q[Q_TT1 * kAlong];
    fc.xxw = q[Q_TT0 * kAlong];
    fc.xye = q[Q_TN1 * kAlong];
    fc.xyw = q[Q_TN0 * kAlong];
    fc.yyn = q[Q_NN1 * kAlong];
    fc.yys = q[Q_NN0 * kAlong];
    fc.yxn = q[Q_NT1 * kAlong];
    fc.yxs = q[Q_NT0 * kAlong];
    const T lphi = lap9f(st, fc, T(g.idx), T(g.idy), i, j, kHX ? RHI : RLO, kHY ? RHI : RLO, b, homog);
    const T newphi = p + (q[Q_F * kAlong] - lphi) * q[Q_D * kAlong];
    S[x[1] + y[1]] = om * newphi + om1 * p;
}

// The sides (bit S_*) whose ghosts follow from three rows of the window beside them, or
// stay as stored (SideLane::put); the others' are filled from phi as a whole.
__device__ __forceinline__ unsigned plain_sides(const BCd& b, int homog) {
    unsigned m = 0;
    bool periodic = false;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        periodic = periodic || b.type[s] == T_PERIODIC;
        if (b.type[s] == T_NEUM || (b.type[s] == T_DIRI && homog && b.mode[s] != M_LAH)) m |= 1u << s;
    }
    return periodic ? 0u : m;
}

// The first sweep's ghosts of a side that is not plain, by the warp of side v (0-3:
// y low, y high, x low, x high), read from pin beside the window's own loads.  (Read
// after them, the far side of a periodic domain was a second round trip to memory and
// a barrier: a sweep of 132 x 140 doubly periodic cells 5.2 -> 4.2 us in FP64, of
// 264 x 280 with one periodic direction 5.5 -> 4.6, of 1024^2 22.2 -> 20.9.)
template <class C, class T>
__device__ __forceinline__ void start_ghosts(T* S, const Window& w, const DFT<T>& pin, const BCd& b, int homog, int nx,
                                             int ny, int v) {
    const bool yside = v < 2, high = v & 1;
    const bool on = v == 0 ? w.yl : v == 1 ? w.yh : v == 2 ? w.xl : w.xh;
    if (!on || (plain_sides(b, homog) >> ((yside ? S_YLO : S_XLO) + (high ? 1 : 0)) & 1u)) return;
    const DFLoadT<T> P{pin};
    const int lo = yside ? (w.xl ? -1 : w.ox) : w.oy, hi = yside ? (w.xh ? nx + 1 : w.wx1) : w.wy1;
    const int side = high ? (yside ? ny : nx) : -1;
    for (int q = lo + (threadIdx.x & 31); q < hi; q += 32) {
        const int i = yside ? q : side, j = yside ? side : q;
        S[x_term<C>(i - w.ox) + y_term<C>(j - w.oy)] = sweep_ghost(P, b, homog, nx, ny, i, j);
    }
}

// What a lane keeps of its side (kY: a y side; kHigh: at the high end, in an odd
// row or column of the window if kOdd).  With the side's parity known, the plane
// places of the sixteen cells a lane reads are constants from one address and the
// two colours whose turns its cells have are too: as registers they were made
// again, some hundred instructions a colour, each time.
template <class C, bool kY, bool kHigh, bool kOdd>
struct SideLane {
    using T = typename C::T;
    static constexpr int sd = (kY ? S_YLO : S_XLO) + (kHigh ? 1 : 0);
    // the colours (0,0),(1,1),(1,0),(0,1): the one with this normal parity and tangential parity c
    __host__ __device__ static constexpr int ph(int c) {
        return kY ? (kOdd ? (c ? 1 : 3) : (c ? 2 : 0)) : (kOdd ? (c ? 1 : 2) : (c ? 3 : 0));
    }
    // Term of row r across the side, at its block (the ghost, the side, one and two inward).
    __host__ __device__ static constexpr int across(int r) {
        constexpr int NQ = kY ? 2 * C::PS : C::PS, NB = kY ? C::P : 1;
        const int low = r == 0 ? NQ - NB : r == 1 ? 0 : r == 2 ? NQ : NB;
        const int odd = r == 0 ? NB : r == 1 ? NQ : r == 2 ? 0 : NQ - NB;
        const int even = r == 0 ? NQ : r == 1 ? 0 : r == 2 ? NQ - NB : -NB;
        return !kHigh ? low : kOdd ? odd : even;
    }
    // Place of column t - 1 of the lane's (its cells are 0 and 1) in row r (the ghost, the side, one and two inward).
    __host__ __device__ static constexpr int at(int t, int r) {
        constexpr int TQ = kY ? C::PS : 2 * C::PS, TB = kY ? 1 : C::P;   // planes and blocks along the side
        return across(r) + (t == 0 ? TQ - TB : t == 1 ? 0 : t == 2 ? TQ : TB);
    }
    // The warp's corner of the domain: (low, low), (high, high), (low, high), (high,
    // low) for y low, y high, x low, x high, so that at most one direction's places
    // depend on the other side's parity (cz).
    static constexpr bool hx = kHigh, hy = kY ? kHigh : !kHigh;
    bool on, plain, neum;      // the window holds the side; its ghosts follow from three rows; a Neumann side
    bool all_plain, any_plain, corner;   // so do every side's, some side's; the window holds the corner and it is to update
    int cz[4];
    bool ok[2], in[2];         // the lane's cells: edge cells to update, cells of the window
    int base;
    // FP64: the operators (Q_*) and the Neumann side's fluxes.  FP32: the weights W_*
    // of the differences to the cell's own value, the operator folded once a call.
    T q[2][11], nb[2];
    T g0[2], g1[2], g2[2];     // what the next sweep's ghosts are made of
    T idt, idn, om, om1;

    __device__ __forceinline__ void place(const Window& w, const GeoT<T>& g, const BCd& b, int homog, int nx, int ny,
                                          T om_, T om1_) {
        const int lane = threadIdx.x & 31;
        on = kY ? (kHigh ? w.yh : w.yl) : (kHigh ? w.xh : w.xl);
        const Per pr = periodic_of(b);
        const bool periodic = kY ? (kHigh ? pr.yh : pr.yl) : (kHigh ? pr.xh : pr.xl);
        const unsigned sides = plain_sides(b, homog);
        plain = sides >> sd & 1u;
        all_plain = sides == 15u;
        any_plain = sides != 0u;
        neum = b.type[sd] == T_NEUM;
        const int ot = kY ? w.ox : w.oy, et = kY ? w.wx1 : w.wy1, nt = kY ? nx : ny;
        const int m = kHigh ? ((kY ? ny - w.oy : nx - w.ox) - 1) >> 1 : 0;   // the side's block, 0 at the low end
        const int lo = (kY ? pr.xl : pr.yl) ? 0 : 1, hi = (kY ? pr.xh : pr.yh) ? nt : nt - 1;   // corners left out
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int t = ot + 2 * lane + c;
            in[c] = on && t < et;
            ok[c] = in[c] && !periodic && t >= lo && t < hi;
        }
        base = C::P + 1 + (kY ? lane + m * C::P : lane * C::P + m);
        corner = lane == 0 && (hx ? w.xh && !pr.xh : w.xl && !pr.xl) && (hy ? w.yh && !pr.yh : w.yl && !pr.yl);
#pragma unroll
        for (int r = 0; r < 4; ++r)   // the direction along the side: the other sides' terms
            cz[r] = kY ? x_term<C>(hx ? nx - 1 - w.ox - (r - 1) : r - 1) : y_term<C>(hy ? ny - 1 - w.oy - (r - 1) : r - 1);
        idt = T(kY ? g.idx : g.idy);
        idn = T(kY ? g.idy : g.idx);
        om = om_;
        om1 = om1_;
    }
    // The operators, once their owners have written the strips.
    __device__ __forceinline__ void take(const T* strips, const Window& w, const BCd& b, int homog) {
        const int lane = threadIdx.x & 31, side = (kY ? 0 : 2) + (kHigh ? 1 : 0);
        const T quarter = T(0.25);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int t = (kY ? w.ox : w.oy) + 2 * lane + c;
            nb[c] = T(0.0);
            if (neum && ok[c]) nb[c] = T(nbval(b, homog, sd, sd == S_YHI ? b.kyhi : t));
            T v[kStrip];
#pragma unroll
            for (int r = 0; r < kStrip; ++r) {
                v[r] = T(0.0);
                if (ok[c]) v[r] = strips[(side * kStrip + r) * kAlong + 2 * lane + c];
                if (r == Q_TN1 || r == Q_TN0 || r == Q_NT1 || r == Q_NT0) v[r] = v[r] * quarter;
            }
            if constexpr (sizeof(T) == 8) {
#pragma unroll
                for (int r = 0; r < kStrip; ++r) q[c][r] = v[r];
            } else {
                // lphi = sum of W (phi - p): the extrapolations are sums of such differences, and the sign s turns the
                // high side's normal inward (in: the face towards the interior, out: the domain's side)
                const T s = kHigh ? T(-1.0) : T(1.0), tt = idt * idt, tn = s * idt * idn, nn = idn * idn;
                const T a1 = v[Q_TT1] * tt, a0 = v[Q_TT0] * tt, b1 = v[Q_TN1] * tn, b0 = v[Q_TN0] * tn;
                const T ci = v[kHigh ? Q_NN0 : Q_NN1] * nn, ei = v[kHigh ? Q_NT0 : Q_NT1] * tn;
                const T co = neum ? T(0.0) : v[kHigh ? Q_NN1 : Q_NN0] * nn;
                const T eo = neum ? T(0.0) : v[kHigh ? Q_NT1 : Q_NT0] * tn;
                q[c][W_PP] = a1 - T(3.0) * b1 + ei - T(4.0) * eo;
                q[c][W_PM] = a0 + T(3.0) * b0 - ei + T(4.0) * eo;
                q[c][W_P1] = T(4.0) * b1 + ei + T(3.0) * eo;
                q[c][W_M1] = -(T(4.0) * b0 + ei + T(3.0) * eo);
                q[c][W_P2] = -(b1 + eo);
                q[c][W_M2] = b0 + eo;
                q[c][W_I1] = T(4.0) * (b1 - b0) + ci;
                q[c][W_I2] = b0 - b1;
                q[c][W_GH] = co;
                q[c][W_D] = v[Q_D] * om;
                q[c][W_F] = v[Q_F] + s * nb[c] * idn;
            }
        }
    }
    // A sweep's ghosts (fill_ghosts without do_neum, P2:1556), of the values at its
    // start.  Where they follow from three rows, grab reads these before the interior
    // colours change them (and may do so before the corners, whose values put reads
    // again) and put writes the ghosts beside the colours, since only the sides' cells
    // read them.  Otherwise start_ghosts and, from the second sweep of a launch on,
    // fill, between barriers.
    __device__ __forceinline__ void grab(const T* S) {
        if (!plain || neum) return;   // a Neumann side's stay as stored
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (in[c]) {
                g0[c] = S[base + at(1 + c, 1)];
                g1[c] = S[base + at(1 + c, 2)];
                g2[c] = S[base + at(1 + c, 3)];
            }
    }
    __device__ __forceinline__ void put(T* S) {
        if (!plain || neum) return;
#pragma unroll
        for (int c = 0; c < 2; ++c) {   // AU:1161-1177, homogeneous
            if (in[c] && !ok[c]) g0[c] = S[base + at(1 + c, 1)];
            if (in[c]) S[base + at(1 + c, 0)] = -(T(3.0) * g0[c]) + g1[c] - T(1.0 / 5.0) * g2[c];
        }
    }
    __device__ __forceinline__ void fill(T* S, const DFT<T>& pin, const Window& w, const BCd& b, int homog, int nx,
                                         int ny) const {
        if (!on || plain || neum) return;
        const StartLoad<C> P{S, w, pin};
        const int lo = kY ? (w.xl ? -1 : w.ox) : w.oy, hi = kY ? (w.xh ? nx + 1 : w.wx1) : w.wy1;
        const int side = kHigh ? (kY ? ny : nx) : -1;
        for (int v = lo + (threadIdx.x & 31); v < hi; v += 32) {
            const int i = kY ? v : side, j = kY ? side : v;
            S[x_term<C>(i - w.ox) + y_term<C>(j - w.oy)] = sweep_ghost(P, b, homog, nx, ny, i, j);
        }
    }
    // gs9's update of the lane's cell c.
    template <int c>
    __device__ __forceinline__ void cell(T* S) const {
        const T three = T(3.0);
        T* B = S + base;
        const T p = B[at(1 + c, 1)], i1 = B[at(1 + c, 2)], i2 = B[at(1 + c, 3)], gh = B[at(1 + c, 0)];
        const T pm = B[at(c, 1)], m1 = B[at(c, 2)], m2 = B[at(c, 3)];
        const T pp = B[at(2 + c, 1)], p1 = B[at(2 + c, 2)], p2 = B[at(2 + c, 3)];
        if constexpr (sizeof(T) == 4) {
            T x = q[c][W_PP] * (pp - p), y = q[c][W_PM] * (pm - p), z = q[c][W_GH] * (gh - p);
            x = __fmaf_rn(q[c][W_P1], p1 - p, x);
            y = __fmaf_rn(q[c][W_M1], m1 - p, y);
            z = __fmaf_rn(q[c][W_I1], i1 - p, z);
            x = __fmaf_rn(q[c][W_P2], p2 - p, x);
            y = __fmaf_rn(q[c][W_M2], m2 - p, y);
            z = __fmaf_rn(q[c][W_I2], i2 - p, z);
            B[at(1 + c, 1)] = __fmaf_rn(q[c][W_F] - ((x + y) + z), q[c][W_D], p);
            return;
        }
        const T x0 = three * (p - i1) + i2, xm = three * (pm - m1) + m2, xp = three * (pp - p1) + p2;
        const T N0 = kHigh ? x0 : i1, S0 = kHigh ? i1 : x0, Np = kHigh ? xp : p1, Sp = kHigh ? p1 : xp;
        const T Nm = kHigh ? xm : m1, Sm = kHigh ? m1 : xm, gn = kHigh ? gh : i1, gs = kHigh ? i1 : gh;
        const T t1 = q[c][Q_TT1] * (pp - p) * idt + q[c][Q_TN1] * (Np - Sp + N0 - S0) * idn;
        const T t0 = q[c][Q_TT0] * (p - pm) * idt + q[c][Q_TN0] * (N0 - S0 + Nm - Sm) * idn;
        T n1 = q[c][Q_NN1] * (gn - p) * idn + q[c][Q_NT1] * (Np - Nm + pp - pm) * idt;
        T n0 = q[c][Q_NN0] * (p - gs) * idn + q[c][Q_NT0] * (pp - pm + Sp - Sm) * idt;
        if (kHigh) n1 = neum ? nb[c] : n1;
        else n0 = neum ? nb[c] : n0;
        const T lphi = (t1 - t0) * idt + (n1 - n0) * idn;
        const T newphi = p + (q[c][Q_F] - lphi) * q[c][Q_D];
        B[at(1 + c, 1)] = om * newphi + om1 * p;
    }
    // The edge cells colour by colour, then the corners, which on a grid of at least
    // 4 x 4 do not read each other.
    template <int kPhase>
    __device__ __forceinline__ void phase(T* S) const {
        if (ph(0) == kPhase) {
            if (ok[0]) cell<0>(S);
        } else if (ph(1) == kPhase) {
            if (ok[1]) cell<1>(S);
        }
        boundary_sync();
    }
    __device__ __forceinline__ void pass(T* S, const T* strips, const Window& w, const GeoT<T>& g, const BCd& b,
                                         int homog, int nx, int ny) {
        phase<0>(S);
        phase<1>(S);
        phase<2>(S);
        phase<3>(S);
        grab(S);   // for the next sweep
        if (corner) {
            const int i = hx ? nx - 1 : 0, j = hy ? ny - 1 : 0;
            T* B = S + base - (kY ? 0 : C::P + 1);   // lane 0's place
            int x[4], y[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                x[r] = kY ? cz[r] : across(r);
                y[r] = kY ? across(r) : cz[r];
            }
            corner_cell<hx, hy>(B, strips + (hy ? kStrip * kAlong : 0) + i - w.ox, x, y, g, b, homog, i, j, om, om1);
        }
    }
};

// Calls f with the side of warp v (0-3: y low, y high, x low, x high) of window w.
template <class C, class F>
__device__ __forceinline__ void with_side(int v, const Window& w, int nx, int ny, F f) {
    if (v == 0) f(SideLane<C, true, false, false>());
    else if (v == 1 && ((ny - 1 - w.oy) & 1)) f(SideLane<C, true, true, true>());
    else if (v == 1) f(SideLane<C, true, true, false>());
    else if (v == 2) f(SideLane<C, false, false, false>());
    else if (v == 3 && ((nx - 1 - w.ox) & 1)) f(SideLane<C, false, true, true>());
    else if (v == 3) f(SideLane<C, false, true, false>());
}

// Ghosts no sweep changes, by warps 0-3: a Neumann side's, as stored, and the
// corners' marker (with a periodic side they are start_ghosts' instead).
template <class C, class T>
__device__ __forceinline__ void fixed_ghosts(T* s, const Window& w, const DFT<T>& pin, const BCd& b, int nx, int ny) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp >= 4) return;
    const bool yside = warp < 2, high = warp & 1;
    const int sd = (warp + 2) & 3;
    const bool on = warp == 0 ? w.yl : warp == 1 ? w.yh : warp == 2 ? w.xl : w.xh;
    const int ot = yside ? w.ox : w.oy, et = yside ? w.wx1 : w.wy1;
    const int at = high ? (yside ? ny : nx) : -1, gt = at - (yside ? w.oy : w.ox);
    if (on && b.type[sd] == T_NEUM) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int a = 2 * lane + c;
            if (ot + a < et) {
                const T v = yside ? AT(pin, ot + a, at) : AT(pin, at, ot + a);
                s[yside ? x_term<C>(a) + y_term<C>(gt) : x_term<C>(gt) + y_term<C>(a)] = v;
            }
        }
    }
    const bool periodic = b.type[S_XLO] == T_PERIODIC || b.type[S_YLO] == T_PERIODIC;
    if (on && yside && !periodic && lane < 2 && (lane ? w.xh : w.xl))
        s[x_term<C>(lane ? nx - w.ox : -1) + y_term<C>(gt)] = bogus<T>();
}

// A freshly loaded block made ready: the sides' strips, the scaled coefficients,
// phi into the planes.  Returns the
// mask of interior cells (bit q: the block's cell q).
template <class C, bool kInner, class T>
__device__ __forceinline__ unsigned settle(Block<T>& k, T* s, T* strips, const Window& w, int kbx, int kby, T idx,
                                           T idy, T om, const BCd& b, int nx, int ny) {
    const int i0 = w.ox + 2 * kbx, j0 = w.oy + 2 * kby;
    if (!kInner && w.any()) {
        const int yh = ny - 1 - j0, xh = nx - 1 - i0;   // the high side's row / column in this block, if 0 or 1
        const int sz = kStrip * kAlong;
        if (w.yl && kby == 0) {
            strip_write<0, 0>(strips + 2 * kbx, k, true);
            strip_write<1, 0>(strips + 2 * kbx + 1, k, true);
        }
        if (w.yh && yh == 0) {
            strip_write<0, 0>(strips + sz + 2 * kbx, k, true);
            strip_write<1, 0>(strips + sz + 2 * kbx + 1, k, true);
        } else if (w.yh && yh == 1) {
            strip_write<0, 1>(strips + sz + 2 * kbx, k, true);
            strip_write<1, 1>(strips + sz + 2 * kbx + 1, k, true);
        }
        if (w.xl && kbx == 0) {
            strip_write<0, 0>(strips + 2 * sz + 2 * kby, k, false);
            strip_write<0, 1>(strips + 2 * sz + 2 * kby + 1, k, false);
        }
        if (w.xh && xh == 0) {
            strip_write<0, 0>(strips + 3 * sz + 2 * kby, k, false);
            strip_write<0, 1>(strips + 3 * sz + 2 * kby + 1, k, false);
        } else if (w.xh && xh == 1) {
            strip_write<1, 0>(strips + 3 * sz + 2 * kby, k, false);
            strip_write<1, 1>(strips + 3 * sz + 2 * kby + 1, k, false);
        }
    }
    const T q = T(0.25);
    if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                k.xy[a][c] = k.xy[a][c] * q;
                k.yx[c][a] = k.yx[c][a] * q;
            }
    } else {
        const T sx = idx * idx, sy = idy * idy, sc = q * idx * idy;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                k.xx[a][c] = k.xx[a][c] * sx;
                k.xy[a][c] = k.xy[a][c] * sc;
                k.yx[c][a] = k.yx[c][a] * sc;
                k.yy[c][a] = k.yy[c][a] * sy;
            }
#pragma unroll
        for (int a = 0; a < 4; ++a) k.d[a >> 1][a & 1] = k.d[a >> 1][a & 1] * om;
    }
    T* own = s + (kby + 1) * C::P + kbx + 1;
    if (kInner) {
#pragma unroll
        for (int c = 0; c < 4; ++c) own[c * C::PS] = k.p[c >> 1][c & 1];
        return 15u;
    }
    const Per pr = periodic_of(b);
    const int mi0 = pr.xl ? 0 : 1, mi1 = pr.xh ? nx : nx - 1;   // interior cells
    const int mj0 = pr.yl ? 0 : 1, mj1 = pr.yh ? ny : ny - 1;
    unsigned mask = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int i = i0 + (c & 1), j = j0 + (c >> 1);
        if (i < w.wx1 && j < w.wy1) own[c * C::PS] = k.p[c >> 1][c & 1];   // past them there may be ghosts
        if (i >= mi0 && i < min(mi1, w.wx1) && j >= mj0 && j < min(mj1, w.wy1)) mask |= 1u << c;
    }
    return mask;
}

// The four interior colours, a CTA barrier after each.
template <class C, class T>
__device__ __forceinline__ void colours(Block<T>& k, T* own, unsigned mask, T idx, T idy, T om, T om1) {
    if (mask & 1u) own[0] = k.p[0][0] = update<C, 0, 0>(k, own, idx, idy, om, om1);
    cta_sync();
    if (mask & 8u) own[3 * C::PS] = k.p[1][1] = update<C, 1, 1>(k, own, idx, idy, om, om1);
    cta_sync();
    if (mask & 2u) own[C::PS] = k.p[0][1] = update<C, 1, 0>(k, own, idx, idy, om, om1);
    cta_sync();
    if (mask & 4u) own[2 * C::PS] = k.p[1][0] = update<C, 0, 1>(k, own, idx, idy, om, om1);
    cta_sync();
}

// phi of the thread's block, as the sides' passes and ghost fills left it.
template <class C, class T>
__device__ __forceinline__ void reload(Block<T>& k, const T* own) {
#pragma unroll
    for (int c = 0; c < 4; ++c) k.p[c >> 1][c & 1] = own[c * C::PS];
}

// The block's cells of the tile, to pout.
template <bool kVec, class T>
__device__ __forceinline__ void store_block(const Block<T>& k, const DFT<T>& pout, const Window& w, int i0, int j0) {
    const bool w0 = i0 >= w.X0 && i0 < w.X1, w1 = w0 && i0 + 1 < w.X1;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = j0 + r;
        if (j < w.Y0 || j >= w.Y1) continue;
        T* o = &AT(pout, i0, j);
        if (kVec && w1) {
            typename Pair<T>::type v;
            v.x = k.p[r][0];
            v.y = k.p[r][1];
            *reinterpret_cast<typename Pair<T>::type*>(o) = v;
        } else {
            if (w0) o[0] = k.p[r][0];
            if (w1) o[1] = k.p[r][1];
        }
    }
}

// The ghost cells next to the tile (the state fill_ghosts leaves: filled at the
// start of the last sweep), by side warp v.
template <class C, class T>
__device__ __forceinline__ void store_ghosts(const T* s, const DFT<T>& pout, const Window& w, int v, int nx, int ny) {
    if (v < 0 || v >= 4) return;
    const bool yside = v < 2;
    if (!(v == 0 ? w.Y0 == 0 : v == 1 ? w.Y1 >= ny : v == 2 ? w.X0 == 0 : w.X1 >= nx)) return;
    const int lo = yside ? (w.X0 == 0 ? -1 : w.X0) : w.Y0, hi = yside ? (w.X1 >= nx ? nx + 1 : w.X1) : w.Y1;
    const int at = v == 0 || v == 2 ? -1 : yside ? ny : nx;
    for (int q = lo + (threadIdx.x & 31); q < hi; q += 32) {
        const int i = yside ? q : at, j = yside ? at : q;
        AT(pout, i, j) = s[x_term<C>(i - w.ox) + y_term<C>(j - w.oy)];
    }
}

// K sweeps of tile (bx, by) of a level's gx x gy tiles, by one CTA of a shape
// with kSep; s and strips are its planes and the sides' strips.  kVec: every
// array's rows are aligned to pairs of elements.  kHeld: the CTA holds the level
// (any memory, its own writes included), so nothing is read as constant or
// ahead of the kernel before.
template <class C, bool kVec, bool kHeld, class T>
__device__ __forceinline__ void sweep_window(T* s, T* strips, const DFT<T>& pin, const DFT<T>& pout, const DFT<T>& rhs,
                                             const DFT<T>& invd, const GeoT<T>& g, const BCd& b, int homog, int nx,
                                             int ny, int gx, int gy, double omega, int K, int bx, int by) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // tile bounds: even, so blocks do not straddle tiles
    const int hx = (nx + 1) >> 1, hy = (ny + 1) >> 1;
    Window w;
    w.set(2 * (bx * hx / gx), min(nx, 2 * ((bx + 1) * hx / gx)), 2 * (by * hy / gy), min(ny, 2 * ((by + 1) * hy / gy)),
          4 * K + 2, 4 * K, 4 * K + 2, 4 * K + 2, nx, ny);
    const bool any_side = w.any();
    const T idx = T(g.idx), idy = T(g.idy), om = T(omega), om1 = T(1.0 - omega);
    if (warp >= C::NI) {   // the counterpart of the blocks' loop below, with the same CTA barriers
        with_side<C>(warp - C::NI, w, nx, ny, [&](auto L) {
            L.place(w, g, b, homog, nx, ny, om, om1);
            if (any_side && !L.all_plain) {
                if (!kHeld) grid_dependency_wait();
                start_ghosts<C>(s, w, pin, b, homog, nx, ny, warp - C::NI);
            }
            cta_sync();   // phi, the strips and these ghosts are in place
            if (any_side && L.any_plain) {
                L.grab(s);
                cta_sync();
            }
            if (any_side) L.take(strips, w, b, homog);
#pragma unroll 1
            for (int sw = 0; sw < K; ++sw) {
                if (any_side) L.put(s);
                for (int c = 0; c < 4; ++c) cta_sync();   // the interior colours
                if (!any_side) continue;
                L.pass(s, strips, w, g, b, homog, nx, ny);
                if (sw + 1 < K && !L.all_plain) {
                    boundary_sync();
                    L.fill(s, pin, w, b, homog, nx, ny);
                }
                cta_sync();
            }
        });
        store_ghosts<C>(s, pout, w, warp - C::NI, nx, ny);
        return;
    }
    const int kbx = threadIdx.x % C::LB, kby = threadIdx.x / C::LB;   // the thread's block
    const bool ahead = kbx == C::LB - 1 || lane == 31;                // its east neighbour is not the next lane's
    const int i0 = w.ox + 2 * kbx, j0 = w.oy + 2 * kby;
    const bool c0 = i0 < w.wx1, c1 = i0 + 1 < w.wx1;
    T* own = s + (kby + 1) * C::P + kbx + 1;
    // 1. the operator, constant during a solve: requested before the wait for
    //    the kernel ahead (the solver launches sweeps as programmatic dependents)
    Block<T> k = {};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = j0 + r;
        const bool in = j < w.wy1;
        const bool f0 = in && i0 <= w.wx1, f1 = in && i0 + 1 <= w.wx1;
        load_pair<kVec, !kHeld>(&AT(g.xx, i0, j), f0, f1, k.xx[r][0], k.xx[r][1]);
        load_pair<kVec, !kHeld>(&AT(g.xy, i0, j), f0, f1, k.xy[r][0], k.xy[r][1]);
        load_pair<kVec, !kHeld>(&AT(invd, i0, j), in && c0, in && c1, k.d[r][0], k.d[r][1]);
        if (ahead && in && c1) {
            k.xx[r][2] = kHeld ? AT(g.xx, i0 + 2, j) : __ldg(&AT(g.xx, i0 + 2, j));
            k.xy[r][2] = kHeld ? AT(g.xy, i0 + 2, j) : __ldg(&AT(g.xy, i0 + 2, j));
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int j = j0 + r;
        const bool in = j <= w.wy1;
        load_pair<kVec, !kHeld>(&AT(g.yy, i0, j), in && c0, in && c1, k.yy[r][0], k.yy[r][1]);
        load_pair<kVec, !kHeld>(&AT(g.yx, i0, j), in && c0, in && c1, k.yx[r][0], k.yx[r][1]);
    }
    if (!kHeld) grid_dependency_wait();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = j0 + r;
        const bool in = j < w.wy1;
        load_pair<kVec, false>(&AT(pin, i0, j), in && c0, in && c1, k.p[r][0], k.p[r][1]);
        load_pair<kVec, false>(&AT(rhs, i0, j), in && c0, in && c1, k.f[r][0], k.f[r][1]);
    }
    if (any_side) fixed_ghosts<C>(s, w, pin, b, nx, ny);
    // a block's east faces are its neighbour lane's west faces
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const T a = __shfl_down_sync(0xffffffffu, k.xx[r][0], 1), c = __shfl_down_sync(0xffffffffu, k.xy[r][0], 1);
        if (!ahead) {
            k.xx[r][2] = a;
            k.xy[r][2] = c;
        }
    }
    const bool grabs = any_side && plain_sides(b, homog) != 0u;   // (not before the loads are on their way)
    const unsigned mask = settle<C, false>(k, s, strips, w, kbx, kby, idx, idy, om, b, nx, ny);
    cta_sync();
    if (grabs) cta_sync();   // 2. the sides' warps have read what the first sweep's ghosts are made of
#pragma unroll 1
    for (int sw = 0; sw < K; ++sw) {
        // the boundary pass of the sweep before changed cells their owners hold
        // in registers, and a block may hold a ghost (an odd side)
        if (any_side) reload<C>(k, own);
        colours<C>(k, own, mask, idx, idy, om, om1);   // 3.
        if (any_side) cta_sync();                      // 4. the sides' cells
    }
    if (any_side) reload<C>(k, own);
    store_block<kVec>(k, pout, w, i0, j0);
}

// FP64 shapes of sixteen warps: windows of 32 x 48, 64 x 24, 40 x 38, 48 x 32 and 52 x 28 cells.
using Small64 = Shape<double, 12, 16, true, 1>;
using Flat64 = Shape<double, 12, 32, true, 1>;
using Square64 = Shape<double, 12, 20, true, 1>;
using Broad64 = Shape<double, 12, 24, true, 1>;
using Wide64 = Shape<double, 12, 26, true, 1>;

}  // namespace

}  // namespace mgp
