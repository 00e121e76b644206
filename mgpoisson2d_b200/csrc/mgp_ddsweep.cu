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

#include "mgp_ddsweep.cuh"
#include "mgp_kernels.cuh"

namespace mgp {

namespace {

template <class T>
using Box2 = DdShape<T, 32>;

template <class T>
__global__ void __launch_bounds__(32 * Box2<T>::NW, 1)
    k_dd_sweep(DFT<T> pin, DFT<T> pout, DFT<T> m, DFT<T> invd, DFT<T> xx, DFT<T> yy, Mirror<T> g, T idx, T idy, int nx,
               int ny, double omega, int K) {
    __shared__ T s[4 * Box2<T>::PS];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    dd_window<Box2<T>, true, false>(s, pin, pout, m, invd, xx, yy, g, idx, idy, nx, ny, gridDim.x, gridDim.y, omega, K,
                                    blockIdx.x, blockIdx.y);
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
    const Mirror<T> mir = mirror_of<T>(b);
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
