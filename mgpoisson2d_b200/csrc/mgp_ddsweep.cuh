// mgp_ddsweep.cuh -- red-black sweeps of the deferred-correction smoother on a
// window of a level by one CTA: the device routine of mgp_ddsweep.cu's kernel,
// which the coarse cycle (mgp_kernels.cu) also runs on the levels it holds.
#pragma once

#include "mgp_kernels.cuh"

namespace mgp {

namespace {

// A CTA's shape: NW warps, LB blocks a row.  (Half the warps and two CTAs an SM
// measured slower at every size: the halo weighs more than the overlap.)
template <class T_, int LB_>
struct DdShape {
    using T = T_;
    static constexpr int NW = sizeof(T) == 4 ? 32 : 16, LB = LB_, RB = 32 / LB;
    static constexpr int WX = 2 * LB, WY = 2 * NW * RB;             // window
    static constexpr int P = LB + 2, PS = P * (NW * RB + 2);        // plane pitch and size, a spare block around
    // largest tile for K sweeps a launch
    static constexpr int tx(int k) { return WX - 4 * k; }
    static constexpr int ty(int k) { return WY - 4 * k; }
};

template <class T>
struct V2;
template <>
struct V2<float> {
    using type = float2;
};
template <>
struct V2<double> {
    using type = double2;
};

// p[0] (if a) and p[1] (if b; b implies a).  kPair: p is aligned to a pair.
template <bool kPair, bool kConst, class T>
__device__ __forceinline__ void get_pair(const T* p, bool a, bool b, T& v0, T& v1) {
    using V = typename V2<T>::type;
    if (kPair && b) {
        const V v = kConst ? __ldg(reinterpret_cast<const V*>(p)) : *reinterpret_cast<const V*>(p);
        v0 = v.x;
        v1 = v.y;
    } else {
        if (a) v0 = kConst ? __ldg(p) : p[0];
        if (b) v1 = kConst ? __ldg(p + 1) : p[1];
    }
}

template <class T>
struct DdBlock {
    T xx[2][3], yy[3][2], d[2][2], m[2][2], p[2][2];   // x-faces [row][face], y-faces [face][column], cells [row][column]
};

// Sides as the sweep sees them: the factor of a cell's own value its ghost has.
template <class T>
struct Mirror {
    T xl, xh, yl, yh;
};

// The update of the block's cell (CX, CY) at (i, j).  kEdge: the cell may lie on
// the domain's sides.  FP64: dd_gs's operations in their order; FP32: the face
// values carry their two grid factors and the inverse diagonal omega.
template <class B, int CX, int CY, bool kEdge, class T>
__device__ __forceinline__ void dd_update(DdBlock<T>& k, T* own, int i, int j, int nx, int ny, const Mirror<T>& g,
                                          T idx, T idy, T om, T om1) {
    const auto N = [&](int dx, int dy) -> T {   // compile-time dx, dy
        const int x = CX + dx, y = CY + dy;
        if (x >= 0 && x <= 1 && y >= 0 && y <= 1) return k.p[y][x];
        return own[((y & 1) * 2 + (x & 1)) * B::PS + (y >> 1) * B::P + (x >> 1)];
    };
    const T p = k.p[CY][CX];
    T pe = N(1, 0), pw = N(-1, 0), pn = N(0, 1), ps = N(0, -1);
    if (kEdge) {
        if (i == 0) pw = g.xl * p;
        if (i == nx - 1) pe = g.xh * p;
        if (j == 0) ps = g.yl * p;
        if (j == ny - 1) pn = g.yh * p;
    }
    T r;
    if constexpr (sizeof(T) == 8) {
        const T xfe = k.xx[CY][CX + 1] * (pe - p) * idx;
        const T xfw = k.xx[CY][CX] * (p - pw) * idx;
        const T yfn = k.yy[CY + 1][CX] * (pn - p) * idy;
        const T yfs = k.yy[CY][CX] * (p - ps) * idy;
        const T lphi = (xfe - xfw) * idx + (yfn - yfs) * idy;
        const T newphi = p + (k.m[CY][CX] - lphi) * k.d[CY][CX];
        r = om * newphi + om1 * p;
    } else {
        T x = k.xx[CY][CX + 1] * (pe - p);
        x = __fmaf_rn(k.xx[CY][CX], pw - p, x);
        T y = k.yy[CY + 1][CX] * (pn - p);
        y = __fmaf_rn(k.yy[CY][CX], ps - p, y);
        r = __fmaf_rn((k.m[CY][CX] - x) - y, k.d[CY][CX], p);
    }
    k.p[CY][CX] = r;
    own[(CY * 2 + CX) * B::PS] = r;
}

// The factors of homogeneous sides (Dirichlet: the ghost is minus the cell; Neumann: the cell).
template <class T>
__device__ __host__ inline Mirror<T> mirror_of(const BCd& b) {
    const auto side = [&](int s) { return b.type[s] == T_DIRI ? T(-1.0) : T(1.0); };
    return Mirror<T>{side(S_XLO), side(S_XHI), side(S_YLO), side(S_YHI)};
}

// K sweeps of tile (bx, by) of a level's gx x gy tiles for the modified rhs m; s
// is the CTA's planes.  kPair: every array's rows are aligned to pairs of
// elements.  kHeld: the CTA holds the level (any memory, its own writes
// included), so nothing is read as constant or ahead of the kernel before.
template <class B, bool kPair, bool kHeld, class T>
__device__ __forceinline__ void dd_window(T* s, const DFT<T>& pin, const DFT<T>& pout, const DFT<T>& m,
                                          const DFT<T>& invd, const DFT<T>& xx, const DFT<T>& yy, const Mirror<T>& g,
                                          T idx, T idy, int nx, int ny, int gx, int gy, double omega, int K, int bx,
                                          int by) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // an even tile of a balanced partition, and its window
    const int hx = (nx + 1) >> 1, hy = (ny + 1) >> 1;
    const int X0 = 2 * (bx * hx / gx), X1 = min(nx, 2 * ((bx + 1) * hx / gx));
    const int Y0 = 2 * (by * hy / gy), Y1 = min(ny, 2 * ((by + 1) * hy / gy));
    const int ox = max(0, X0 - 2 * K), wx1 = min(nx, X1 + 2 * K);
    const int oy = max(0, Y0 - 2 * K), wy1 = min(ny, Y1 + 2 * K);
    const bool edge = ox == 0 || oy == 0 || wx1 == nx || wy1 == ny;
    const int kbx = lane % B::LB, kby = warp * B::RB + lane / B::LB;   // the thread's block
    const int i0 = ox + 2 * kbx, j0 = oy + 2 * kby;
    const bool c0 = i0 < wx1, c1 = i0 + 1 < wx1;
    T* own = s + (kby + 1) * B::P + kbx + 1;
    DdBlock<T> k = {};
    // what no kernel ahead writes
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool in = j0 + r < wy1;
        get_pair<kPair, !kHeld>(&AT(xx, i0, j0 + r), in && i0 <= wx1, in && i0 + 1 <= wx1, k.xx[r][0], k.xx[r][1]);
        get_pair<kPair, !kHeld>(&AT(invd, i0, j0 + r), in && c0, in && c1, k.d[r][0], k.d[r][1]);
        if (kbx == B::LB - 1 && in && c1) k.xx[r][2] = kHeld ? AT(xx, i0 + 2, j0 + r) : __ldg(&AT(xx, i0 + 2, j0 + r));
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const bool in = j0 + r <= wy1;
        get_pair<kPair, !kHeld>(&AT(yy, i0, j0 + r), in && c0, in && c1, k.yy[r][0], k.yy[r][1]);
    }
    if (!kHeld) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool in = j0 + r < wy1;
        get_pair<kPair, false>(&AT(pin, i0, j0 + r), in && c0, in && c1, k.p[r][0], k.p[r][1]);
        get_pair<kPair, false>(&AT(m, i0, j0 + r), in && c0, in && c1, k.m[r][0], k.m[r][1]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {   // the block's east face is its neighbour's west face
        const T a = __shfl_down_sync(0xffffffffu, k.xx[r][0], 1);
        if (kbx < B::LB - 1) k.xx[r][2] = a;
    }
    const T om = T(omega), om1 = T(1.0 - omega);
    if constexpr (sizeof(T) == 4) {
        const T sx = idx * idx, sy = idy * idy;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                k.xx[a][c] = k.xx[a][c] * sx;
                k.yy[c][a] = k.yy[c][a] * sy;
            }
#pragma unroll
        for (int a = 0; a < 4; ++a) k.d[a >> 1][a & 1] = k.d[a >> 1][a & 1] * om;
    }
    unsigned mask = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        own[q * B::PS] = k.p[q >> 1][q & 1];
        if (i0 + (q & 1) < wx1 && j0 + (q >> 1) < wy1) mask |= 1u << q;
    }
    __syncthreads();
    T before[2][2];   // the block at the start of the last sweep: what its ghosts mirror
    if (edge) {
#pragma unroll 1
        for (int sw = 0; sw < K; ++sw) {
#pragma unroll
            for (int q = 0; q < 4; ++q) before[q >> 1][q & 1] = k.p[q >> 1][q & 1];
            if (mask & 1u) dd_update<B, 0, 0, true>(k, own, i0, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 8u) dd_update<B, 1, 1, true>(k, own, i0 + 1, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
            if (mask & 2u) dd_update<B, 1, 0, true>(k, own, i0 + 1, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 4u) dd_update<B, 0, 1, true>(k, own, i0, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
        }
    } else {
#pragma unroll 1
        for (int sw = 0; sw < K; ++sw) {
            if (mask & 1u) dd_update<B, 0, 0, false>(k, own, i0, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 8u) dd_update<B, 1, 1, false>(k, own, i0 + 1, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
            if (mask & 2u) dd_update<B, 1, 0, false>(k, own, i0 + 1, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 4u) dd_update<B, 0, 1, false>(k, own, i0, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
        }
    }
    const bool w0 = i0 >= X0 && i0 < X1, w1 = w0 && i0 + 1 < X1;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = j0 + r;
        if (j < Y0 || j >= Y1) continue;
        T* o = &AT(pout, i0, j);
        if (kPair && w1) {
            typename V2<T>::type v;
            v.x = k.p[r][0];
            v.y = k.p[r][1];
            *reinterpret_cast<typename V2<T>::type*>(o) = v;
        } else {
            if (w0) o[0] = k.p[r][0];
            if (w1) o[1] = k.p[r][1];
        }
    }
    if (!edge) return;
    // the ghosts the last sweep's fill left (LAH, AU:1277-1492)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = i0 + (q & 1), j = j0 + (q >> 1);
        if (i < X0 || i >= X1 || j < Y0 || j >= Y1) continue;
        const T b = before[q >> 1][q & 1];
        if (i == 0) AT(pout, -1, j) = g.xl * b;
        if (i == nx - 1) AT(pout, nx, j) = g.xh * b;
        if (j == 0) AT(pout, i, -1) = g.yl * b;
        if (j == ny - 1) AT(pout, i, ny) = g.yh * b;
        if ((i == 0 || i == nx - 1) && (j == 0 || j == ny - 1))
            AT(pout, i ? nx : -1, j ? ny : -1) = bogus<T>();
    }
}

}  // namespace

}  // namespace mgp
