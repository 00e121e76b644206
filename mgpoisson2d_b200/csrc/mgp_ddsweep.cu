// mgp_ddsweep.cu -- red-black sweeps of the deferred-correction smoother
// (DD:153-334), several per launch.
//
// The DD smoother is a 5-point Gauss-Seidel sweep on a modified right-hand side
// that stays fixed during a smoothing call, with ghosts refilled at the start of
// each sweep (DD:259): minus the cell beside a Dirichlet side, the cell itself
// beside a Neumann side.  A cell is updated once a sweep and its ghost depends
// on nothing else, so at its update the ghost is -p or p of its own value and
// no ghost is stored.
//
// As three launches a sweep (ghosts, red, black) a 256^2 FP32 level took 5.3 us of
// launch latency a sweep, and a 2048^2 one read every operand twice, since a
// colour touches every line: 22.4 us (now 1.2 and 15.2).  Here a CTA makes K sweeps of a tile: a
// colour reaches one cell, so the window is the tile and 2 K cells around it;
// every pass runs on the whole window, and what it gets wrong at the rim moves
// inward one cell a pass, never into the tile.  The operator is in registers: a
// thread owns a 2 x 2 block (two cells of each colour) with its faces, inverse
// diagonals and modified right-hand side; shared memory holds phi as four parity
// planes, so neighbour reads are consecutive words.  A launch reads phi from one
// buffer and writes the other.
#include <algorithm>
#include <mutex>

#include "mgp_kernels.cuh"

namespace mgp {

namespace {

// A CTA's shape: NW warps, a row of 32 blocks each.  (Half the warps and two CTAs
// an SM measured slower at every size: the halo weighs more than the overlap.)
template <class T>
struct Box2 {
    static constexpr int NW = sizeof(T) == 4 ? 32 : 16;
    static constexpr int WX = 64, WY = 2 * NW;            // window
    static constexpr int P = 34, PS = P * (NW + 2);       // plane pitch and size, a spare block around
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

// p[0] (if a) and p[1] (if b; b implies a); p is aligned to a pair.
template <bool kConst, class T>
__device__ __forceinline__ void get_pair(const T* p, bool a, bool b, T& v0, T& v1) {
    using V = typename V2<T>::type;
    if (b) {
        const V v = kConst ? __ldg(reinterpret_cast<const V*>(p)) : *reinterpret_cast<const V*>(p);
        v0 = v.x;
        v1 = v.y;
    } else if (a) {
        v0 = kConst ? __ldg(p) : p[0];
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
template <int CX, int CY, bool kEdge, class T>
__device__ __forceinline__ void dd_update(DdBlock<T>& k, T* own, int i, int j, int nx, int ny, const Mirror<T>& g,
                                          T idx, T idy, T om, T om1) {
    using B = Box2<T>;
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

template <class T>
__global__ void __launch_bounds__(32 * Box2<T>::NW, 1)
    k_dd_sweep(DFT<T> pin, DFT<T> pout, DFT<T> m, DFT<T> invd, DFT<T> xx, DFT<T> yy, Mirror<T> g, T idx, T idy, int nx,
               int ny, double omega, int K) {
    using B = Box2<T>;
    __shared__ T s[4 * B::PS];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // an even tile of a balanced partition, and its window
    const int hx = (nx + 1) >> 1, hy = (ny + 1) >> 1, gx = gridDim.x, gy = gridDim.y;
    const int X0 = 2 * ((int)blockIdx.x * hx / gx), X1 = min(nx, 2 * (((int)blockIdx.x + 1) * hx / gx));
    const int Y0 = 2 * ((int)blockIdx.y * hy / gy), Y1 = min(ny, 2 * (((int)blockIdx.y + 1) * hy / gy));
    const int ox = max(0, X0 - 2 * K), wx1 = min(nx, X1 + 2 * K);
    const int oy = max(0, Y0 - 2 * K), wy1 = min(ny, Y1 + 2 * K);
    const bool edge = ox == 0 || oy == 0 || wx1 == nx || wy1 == ny;
    const int i0 = ox + 2 * lane, j0 = oy + 2 * warp;
    const bool c0 = i0 < wx1, c1 = i0 + 1 < wx1;
    T* own = s + (warp + 1) * B::P + lane + 1;
    DdBlock<T> k = {};
    // what no kernel ahead writes
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool in = j0 + r < wy1;
        get_pair<true>(&AT(xx, i0, j0 + r), in && i0 <= wx1, in && i0 + 1 <= wx1, k.xx[r][0], k.xx[r][1]);
        get_pair<true>(&AT(invd, i0, j0 + r), in && c0, in && c1, k.d[r][0], k.d[r][1]);
        if (lane == 31 && in && c1) k.xx[r][2] = __ldg(&AT(xx, i0 + 2, j0 + r));
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const bool in = j0 + r <= wy1;
        get_pair<true>(&AT(yy, i0, j0 + r), in && c0, in && c1, k.yy[r][0], k.yy[r][1]);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool in = j0 + r < wy1;
        get_pair<false>(&AT(pin, i0, j0 + r), in && c0, in && c1, k.p[r][0], k.p[r][1]);
        get_pair<false>(&AT(m, i0, j0 + r), in && c0, in && c1, k.m[r][0], k.m[r][1]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {   // the block's east face is its neighbour's west face
        const T a = __shfl_down_sync(0xffffffffu, k.xx[r][0], 1);
        if (lane < 31) k.xx[r][2] = a;
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
            if (mask & 1u) dd_update<0, 0, true>(k, own, i0, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 8u) dd_update<1, 1, true>(k, own, i0 + 1, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
            if (mask & 2u) dd_update<1, 0, true>(k, own, i0 + 1, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 4u) dd_update<0, 1, true>(k, own, i0, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
        }
    } else {
#pragma unroll 1
        for (int sw = 0; sw < K; ++sw) {
            if (mask & 1u) dd_update<0, 0, false>(k, own, i0, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 8u) dd_update<1, 1, false>(k, own, i0 + 1, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
            if (mask & 2u) dd_update<1, 0, false>(k, own, i0 + 1, j0, nx, ny, g, idx, idy, om, om1);
            if (mask & 4u) dd_update<0, 1, false>(k, own, i0, j0 + 1, nx, ny, g, idx, idy, om, om1);
            __syncthreads();
        }
    }
    const bool w0 = i0 >= X0 && i0 < X1, w1 = w0 && i0 + 1 < X1;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = j0 + r;
        if (j < Y0 || j >= Y1) continue;
        T* o = &AT(pout, i0, j);
        if (w1) {
            typename V2<T>::type v;
            v.x = k.p[r][0];
            v.y = k.p[r][1];
            *reinterpret_cast<typename V2<T>::type*>(o) = v;
        } else if (w0) {
            o[0] = k.p[r][0];
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

int sms() {
    static std::mutex mu;
    static int n[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    std::lock_guard<std::mutex> lock(mu);
    if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        n[dev] = 148;
    }
    return n[dev];
}

template <class T>
bool pairs(const DFT<T>& f) {
    return (reinterpret_cast<uintptr_t>(f.p) & (2 * sizeof(T) - 1)) == 0 && (f.ld & 1) == 0;
}

template <class B>
long tiles(int nx, int ny, int k, int* gx, int* gy) {
    if (k < 1 || B::tx(k) < 2 || B::ty(k) < 2) return 1L << 40;
    *gx = nx <= B::WX ? 1 : ((nx + 1) / 2 + B::tx(k) / 2 - 1) / (B::tx(k) / 2);
    *gy = ny <= B::WY ? 1 : ((ny + 1) / 2 + B::ty(k) / 2 - 1) / (B::ty(k) / 2);
    return (long)*gx * *gy;
}

// Sweeps of the next launch, of `left` still to do (0: the caller's launch per
// colour is faster).  A level one window holds takes all of them; else the most
// of 4 and 2 whose tiles do not outnumber the SMs, since such a launch lasts one
// CTA's latency; a larger level takes 4, or the 2 or 3 that are left.  us a sweep,
// FP32 / FP64, for 4, 2, 1 a launch and for a launch per colour: 256^2 1.2, 1.9,
// 3.2, 5.3 / 1.3, 1.9, 3.1, 5.6; 1024^2 4.5, 5.8, 10.3, 9.1 / 10.9, 10.7, 15.1,
// 11.8; 2048^2 15.2, 20.4, 38.8, 22.4 / 41.0, 41.7, 73.5, 62.5: one sweep a
// launch pays only while its tiles are about the SMs.
template <class B>
int dd_sweeps_now(int nx, int ny, int left, int* gx, int* gy) {
    int k = left;
    if (nx > B::WX || ny > B::WY) {
        k = std::min(left, 4);
        if (k >= 2 && tiles<B>(nx, ny, k, gx, gy) > sms() && tiles<B>(nx, ny, 2, gx, gy) <= sms()) k = 2;
        if (k == 1 && 2 * tiles<B>(nx, ny, 1, gx, gy) > 3 * sms()) return 0;
    }
    tiles<B>(nx, ny, k, gx, gy);
    return k;
}

template <class T>
cudaError_t dd_sweep_impl(const DFT<T>& pin, const DFT<T>& pout, const DFT<T>& m, const DFT<T>& invd,
                          const GeoT<T>& g, const BCd& b, int nx, int ny, double omega, int left, int* done,
                          cudaStream_t st) {
    using B = Box2<T>;
    if (!pairs(pin) || !pairs(pout) || !pairs(m) || !pairs(invd) || !pairs(g.xx) || !pairs(g.yy))
        return cudaErrorMisalignedAddress;
    int gx = 1, gy = 1;
    *done = dd_sweeps_now<B>(nx, ny, left, &gx, &gy);
    if (!*done) return cudaSuccess;
    const auto side = [&](int s) { return b.type[s] == T_DIRI ? T(-1.0) : T(1.0); };
    const Mirror<T> mir{side(S_XLO), side(S_XHI), side(S_YLO), side(S_YHI)};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gx, gy);
    cfg.blockDim = dim3(32 * B::NW);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, k_dd_sweep<T>, pin, pout, m, invd, g.xx, g.yy, mir, T(g.idx), T(g.idy), nx, ny,
                              omega, *done);
}

}  // namespace

bool dd_sweep_fusable(const BCd& b) {
    for (int s = 0; s < 4; ++s)
        if ((b.type[s] != T_DIRI && b.type[s] != T_NEUM) || b.mode[s] != M_LAH) return false;
    return true;
}

cudaError_t launch_dd_sweeps(const DF& pin, const DF& pout, const DF& m, const DF& invd, const Geo& g, const BCd& b,
                             int nx, int ny, double omega, int left, int* done, cudaStream_t st) {
    return dd_sweep_impl(pin, pout, m, invd, g, b, nx, ny, omega, left, done, st);
}
cudaError_t launch_dd_sweeps(const DF32& pin, const DF32& pout, const DF32& m, const DF32& invd, const Geo32& g,
                             const BCd& b, int nx, int ny, double omega, int left, int* done, cudaStream_t st) {
    return dd_sweep_impl(pin, pout, m, invd, g, b, nx, ny, omega, left, done, st);
}

}  // namespace mgp
