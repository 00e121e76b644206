// The exact bottom of hierarchies whose schedule stops above kDirectLargeCells
// cells (an odd side), by block cyclic reduction.
//
// The level's B lines of m cells (m the shorter side) make its operator block
// tridiagonal: a line's equations reach one line to either side, the first and
// last line's two.  A step of the reduction eliminates every second line that is
// left, so a solve is 2 log2(B) + 1 dependent steps, each a set of independent
// dense m x m matrix-vector products: 5 B m^2 doubles read once.  solve_bicgstab2
// on such a level was some five thousand barrier-separated phases of one cluster,
// 10.3 ms on 105 x 54 cells whatever the chip; the reduction's 15 launches take
// 33 us there, most of it their latency (12 MB of factors).  FP64 throughout, partial pivoting
// inside the blocks; the factorisation is kept only if it solves (k_bb_check).
#include <algorithm>
#include <vector>

#include "mgp_kernels.cuh"

namespace mgp {

namespace {

constexpr int kRowThreads = 256;               // a warp per row of a block
constexpr int kRowsPerCta = kRowThreads / 32;
constexpr int kVec = (kBlockLineMax + 31) / 32;   // a lane's share of a row

__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_allow() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A row of a block: a lane's elements (zero where the block is absent).
__device__ __forceinline__ void row_load(double* f, const double* row, bool there, int m, int lane) {
#pragma unroll
    for (int q = 0; q < kVec; ++q) f[q] = (there && lane + 32 * q < m) ? __ldg(row + lane + 32 * q) : 0.0;
}
// acc + row . v
__device__ __forceinline__ double row_dot(double acc, const double* f, const double* v, long stride, bool there, int m,
                                          int lane) {
    if (!there) return acc;
#pragma unroll
    for (int q = 0; q < kVec; ++q)
        if (lane + 32 * q < m) acc = acc + f[q] * v[(lane + 32 * q) * stride];
    return acc;
}
__device__ __forceinline__ double row_sum(double s) {
    for (int o = 16; o > 0; o >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// One step down: the lines that stay take up their eliminated neighbours,
// r_p -= F r_l + G r_r.  item: line, eliminated neighbours (-1: none), F's index.
// The factors do not depend on the step ahead: they are read before the wait.
__device__ __forceinline__ void step_down(const BlockBottom& b, const DF& r, int first, int4 it, int row) {
    const int lane = threadIdx.x & 31, m = b.m;
    const double* F = b.fg + ((long)it.w * m + row) * m;
    double f[kVec], g[kVec];
    const bool here = row < m;
    row_load(f, F, here && it.y >= 0, m, lane);
    row_load(g, F + (long)m * m, here && it.z >= 0, m, lane);
    dep_allow();
    dep_wait();
    if (!here) return;
    const double* v = first ? r.p : b.r;
    const long sl = first ? (b.along_y ? (long)r.ld : 1) : m, sc = first ? (b.along_y ? 1 : (long)r.ld) : 1;
    const double own = v[it.x * sl + row * sc];
    double s = row_dot(0.0, f, v + it.y * sl, sc, it.y >= 0, m, lane);
    s = row_sum(row_dot(s, g, v + it.z * sl, sc, it.z >= 0, m, lane));
    if (lane == 0) b.r[(long)it.x * m + row] = own - s;
}

// One step up: the eliminated lines from their neighbours, x_p = D^-1 r_p - P x_l - Q x_r.
__device__ __forceinline__ void step_up(const BlockBottom& b, const DF& e, const DF& r, int first, int4 it, int row) {
    const int lane = threadIdx.x & 31, m = b.m;
    const long o = ((long)it.x * m + row) * m;
    double d[kVec], p[kVec], q[kVec];
    const bool here = row < m;
    row_load(d, b.dinv + o, here, m, lane);
    row_load(p, b.p + o, here && it.y >= 0, m, lane);
    row_load(q, b.q + o, here && it.z >= 0, m, lane);
    dep_allow();
    dep_wait();
    if (!here) return;
    const double* v = first ? r.p : b.r;
    const long sl = first ? (b.along_y ? (long)r.ld : 1) : m, sc = first ? (b.along_y ? 1 : (long)r.ld) : 1;
    const long el = b.along_y ? (long)e.ld : 1, ec = b.along_y ? 1 : (long)e.ld;
    const double t = row_dot(0.0, d, v + it.x * sl, sc, true, m, lane);
    double s = row_dot(0.0, p, e.p + it.y * el, ec, it.y >= 0, m, lane);
    s = row_dot(s, q, e.p + it.z * el, ec, it.z >= 0, m, lane);
    const double x = row_sum(t - s);
    if (lane == 0) e.p[it.x * el + row * ec] = x;
}

__global__ void __launch_bounds__(kRowThreads) k_bb_down(BlockBottom b, DF r, int first, const int4* __restrict__ items) {
    step_down(b, r, first, __ldg(items + blockIdx.y), blockIdx.x * kRowsPerCta + (threadIdx.x >> 5));
}
__global__ void __launch_bounds__(kRowThreads) k_bb_up(BlockBottom b, DF e, DF r, int first,
                                                       const int4* __restrict__ items) {
    step_up(b, e, r, first, __ldg(items + blockIdx.y), blockIdx.x * kRowsPerCta + (threadIdx.x >> 5));
}

// Step l of many problems (lockstep batches): job k owns blocks [pre[k], pre[k + 1]),
// none where its reduction has fewer steps.  The factors and the tables do not
// depend on the launch ahead.
template <bool kUp>
__global__ void __launch_bounds__(kRowThreads) k_bb_jobs(const BlockJob* __restrict__ jobs, const int* __restrict__ pre,
                                                         int njobs, int l) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {   // the last job with pre[job] <= the block
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(pre + mid) <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const BlockJob& J = jobs[lo];
    const int rows = (J.b.m + kRowsPerCta - 1) / kRowsPerCta, q = blockIdx.x - __ldg(pre + lo);
    const int4 it = __ldg(J.b.items + (kUp ? J.b.oup[l] : J.b.odown[l]) + q / rows);
    const int row = (q % rows) * kRowsPerCta + (threadIdx.x >> 5);
    if (kUp) step_up(J.b, J.e, J.r, l == 0, it, row);
    else step_down(J.b, J.r, l == 0, it, row);
}

template <class... KArgs, class... Args>
cudaError_t launch_step(void (*k)(KArgs...), dim3 grid, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kRowThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, k, std::forward<Args>(args)...);
}

// ---------------------------------------------------------------------------
// Set-up
// ---------------------------------------------------------------------------
// The operator's entries by probing: cells five apart along each axis have
// disjoint supports (reach two), so a field of ones on one colour gives a column
// of every cell of that colour at once.  Along a periodic axis the cells past the
// last whole five take colours of their own.
__host__ __device__ inline int probe_colour(int c, int n, bool periodic) {
    const int whole = n - n % 5;
    return (periodic && c >= whole) ? 5 + c - whole : c % 5;
}
inline int probe_colours(int n, bool periodic) { return 5 + (periodic ? n % 5 : 0); }

__global__ void k_bb_probe(DF phi, int nx, int ny, int px, int py, int cx, int cy) {
    const int i = (int)(blockIdx.x * 32 + threadIdx.x) - 1, j = (int)(blockIdx.y * 8 + threadIdx.y) - 1;
    if (i > nx || j > ny) return;
    const bool in = i >= 0 && i < nx && j >= 0 && j < ny;
    phi.p[(long)j * phi.ld + i] =
        (in && probe_colour(i, nx, px) == cx && probe_colour(j, ny, py) == cy) ? 1.0 : 0.0;
}

// The blocks of line blockIdx.x: D, A (line before), C (line after) and e0, e1
// (two lines on from the first, two back from the last).  All zero before.
__global__ void k_bb_gather(const double* out, size_t field, int ld, int along_y, int m, int B, int pc, int ncc, int ncl,
                            double* D, double* A, double* C, double* e0, double* e1) {
    const int line = blockIdx.x;
    const long mm = (long)m * m;
    for (int k = threadIdx.x; k < 25 * m; k += blockDim.x) {
        const int row = k / 25, dl = (k % 25) / 5 - 2, l = line + dl;
        int c = row + k % 5 - 2;
        if (pc) c = (c + m) % m;
        if (l < 0 || l >= B || c < 0 || c >= m) continue;
        const int qc = probe_colour(c, m, pc), ql = probe_colour(l, B, false);
        const double* f = out + field * (size_t)(ql * ncc + qc) + ld + 1;
        const double v = along_y ? f[(long)line * ld + row] : f[(long)row * ld + line];
        double* to = dl == 0 ? D + line * mm : dl == -1 ? A + line * mm : dl == 1 ? C + line * mm
                     : (dl == 2 && line == 0) ? e0 : (dl == -2 && line == B - 1) ? e1 : nullptr;
        if (to) to[(long)row * m + c] = v;
    }
}

// In-place Gauss-Jordan inversion with row pivoting, a block per CTA in shared memory.
constexpr int kInvThreads = 1024;
__global__ void __launch_bounds__(kInvThreads) k_bb_invert(double* D, const int4* __restrict__ items, int m, int* fail) {
    extern __shared__ double a[];
    __shared__ int perm[kBlockLineMax];
    __shared__ double col[kBlockLineMax];
    __shared__ double s_p;
    const int ld = m | 1, t = threadIdx.x, tx = t & 31, ty = t >> 5;
    double* M = D + (long)items[blockIdx.x].x * m * m;
    for (int i = ty; i < m; i += 32)
        for (int j = tx; j < m; j += 32) a[i * ld + j] = M[(long)i * m + j];
    __syncthreads();
    for (int k = 0; k < m; ++k) {
        if (ty == 0) {
            double best = -1.0;
            int at = k;
            for (int i = k + tx; i < m; i += 32) {
                const double v = fabs(a[i * ld + k]);
                if (v > best) {
                    best = v;
                    at = i;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double v = __shfl_xor_sync(0xffffffffu, best, o);
                const int w = __shfl_xor_sync(0xffffffffu, at, o);
                if (v > best || (v == best && w < at)) {
                    best = v;
                    at = w;
                }
            }
            if (tx == 0) {
                perm[k] = at;
                s_p = 1.0 / a[at * ld + k];
                if (!(best > 0.0) || !isfinite(best)) *fail = 1;
            }
        }
        __syncthreads();
        const int pr = perm[k];
        const double p = s_p;
        if (t < m && t != k) {
            const double vk = a[k * ld + t], vp = a[pr * ld + t];
            a[pr * ld + t] = vk;
            a[k * ld + t] = vp * p;
        }
        if (t >= 512 && t - 512 < m) col[t - 512] = (t - 512 == pr) ? a[k * ld + k] : a[(t - 512) * ld + k];
        __syncthreads();
        for (int i = ty; i < m; i += 32) {
            if (i == k) {
                if (tx == 0) a[k * ld + k] = p;
                continue;
            }
            const double f = col[i];
            for (int j = tx; j < m; j += 32)
                a[i * ld + j] = (j == k) ? -f * p : a[i * ld + j] - f * a[k * ld + j];
        }
        __syncthreads();
    }
    if (t < m)
        for (int k = m - 1; k >= 0; --k)
            if (perm[k] != k) {
                const double x = a[t * ld + k];
                a[t * ld + k] = a[t * ld + perm[k]];
                a[t * ld + perm[k]] = x;
            }
    __syncthreads();
    for (int i = ty; i < m; i += 32)
        for (int j = tx; j < m; j += 32) M[(long)i * m + j] = a[i * ld + j];
}

// c = c0 + s (a1 b1 + a2 b2), m x m each; c0, a1 and a2 may be null.
struct BlockMul {
    double* c;
    const double *c0, *a1, *b1, *a2, *b2;
    double s;
};
__global__ void __launch_bounds__(256) k_bb_mul(const BlockMul* __restrict__ jobs, int m) {
    __shared__ double sa[32][17], sb[16][33];
    const BlockMul J = jobs[blockIdx.y];
    const int tiles = (m + 31) / 32, i0 = (blockIdx.x / tiles) * 32, j0 = (blockIdx.x % tiles) * 32;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[2][2] = {{0, 0}, {0, 0}};
    for (int q = 0; q < 2; ++q) {
        const double *A = q ? J.a2 : J.a1, *Bm = q ? J.b2 : J.b1;
        if (!A) continue;
        for (int k0 = 0; k0 < m; k0 += 16) {
            for (int k = threadIdx.x; k < 512; k += 256) {
                const int i = i0 + k / 16, kk = k0 + k % 16, kb = k0 + k / 32, j = j0 + k % 32;
                sa[k / 16][k % 16] = (i < m && kk < m) ? A[(long)i * m + kk] : 0.0;
                sb[k / 32][k % 32] = (kb < m && j < m) ? Bm[(long)kb * m + j] : 0.0;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const double x0 = sa[ty][k], x1 = sa[ty + 16][k], y0 = sb[k][tx], y1 = sb[k][tx + 16];
                acc[0][0] += x0 * y0;
                acc[0][1] += x0 * y1;
                acc[1][0] += x1 * y0;
                acc[1][1] += x1 * y1;
            }
            __syncthreads();
        }
    }
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v) {
            const int i = i0 + ty + 16 * u, j = j0 + tx + 16 * v;
            if (i < m && j < m) {
                const long o = (long)i * m + j;
                J.c[o] = (J.c0 ? J.c0[o] : 0.0) + J.s * acc[u][v];
            }
        }
}

// A right-hand side of independent signs, and the test of its solution: the
// bottom this replaces stops at 1e-6 of its first residual.
__global__ void k_bb_rhs(DF r, int nx, int ny) {
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
    if (i >= nx || j >= ny) return;
    unsigned h = (unsigned)(j * nx + i) * 2654435761u + 12345u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    r.p[(long)j * r.ld + i] = (h & 1) ? 1.0 : -1.0;
}
__global__ void __launch_bounds__(1024) k_bb_check(DF res, int nx, int ny, int* fail) {
    bool bad = false;
    for (long k = threadIdx.x; k < (long)nx * ny; k += blockDim.x)
        bad = bad || !(fabs(res.p[(k / nx) * res.ld + k % nx]) <= 1e-8);
    if (bad) *fail = 1;
}

struct Step {
    std::vector<int4> down, up;
    std::vector<BlockMul> first, second;
};

// The order of elimination of B lines.
std::vector<Step> elimination(int B) {
    std::vector<Step> steps;
    std::vector<int> act(B);
    for (int k = 0; k < B; ++k) act[k] = k;
    int nfg = 0;
    while (act.size() > 1) {
        const int n = (int)act.size();
        std::vector<char> gone(n, 0);
        for (int k = 1; k < n; k += 2) gone[k] = 1;
        if (steps.empty() && n % 2 == 0) {   // lines 1 and n - 2 go first: their neighbours reach past them
            gone[n - 3] = gone[n - 1] = 0;
            gone[n - 2] = 1;
        }
        Step s;
        std::vector<int> keep;
        for (int k = 0; k < n; ++k) {
            const int l = k > 0 ? act[k - 1] : -1, r = k + 1 < n ? act[k + 1] : -1;
            if (gone[k]) {
                s.up.push_back(int4{act[k], l, r, 0});
            } else {
                s.down.push_back(int4{act[k], (k > 0 && gone[k - 1]) ? l : -1, (k + 1 < n && gone[k + 1]) ? r : -1, nfg});
                nfg += 2;
                keep.push_back(act[k]);
            }
        }
        steps.push_back(s);
        act = keep;
    }
    return steps;
}

// Doubles of memory: what the solves read (keep), and the set-up's own (temp).
struct Sizes {
    int nfg, nc, nl, np;   // blocks of F and G; probing colours across and along the lines, and fields
    bool pc;               // the lines close on themselves
    size_t ld, field, keep, temp;
    Sizes(const BlockBottom& b, int nx, int ny, bool px, bool py) {
        const size_t mm = (size_t)b.m * b.m;
        nfg = 0;
        for (const Step& s : elimination(b.lines)) nfg += 2 * (int)s.down.size();
        pc = b.along_y ? px : py;
        nc = probe_colours(b.m, pc);
        nl = probe_colours(b.lines, false);
        np = nc * nl;
        ld = nx + 2;
        field = ld * (ny + 2);
        keep = (size_t)(3 * b.lines + nfg) * mm + (size_t)b.lines * b.m;
        temp = (size_t)(2 * b.lines + 2) * mm + (size_t)(np + 3) * field;
    }
};

}  // namespace

bool block_bottom_shape(int nx, int ny, const BCd& bc, BlockBottom* b) {
    for (int k = 0; k < 4; ++k)
        if (bc.type[k] != T_DIRI && bc.type[k] != T_NEUM && bc.type[k] != T_PERIODIC) return false;
    const bool px = bc.type[0] == T_PERIODIC, py = bc.type[2] == T_PERIODIC;
    if ((px && py) || px != (bc.type[1] == T_PERIODIC) || py != (bc.type[3] == T_PERIODIC)) return false;
    b->along_y = px ? 1 : py ? 0 : nx <= ny;
    b->m = b->along_y ? nx : ny;
    b->lines = b->along_y ? ny : nx;
    // (lines: a launch has a block of the grid's second dimension per product, at most two a line)
    return b->m >= 5 && b->lines >= 6 && b->m <= kBlockLineMax && b->lines <= kBlockLinesMax &&
           5.0 * b->lines * b->m * b->m * sizeof(double) <= (double)kBlockBytesMax;
}

size_t block_bottom_peak_bytes(int nx, int ny, const BCd& bc) {
    BlockBottom b = {};
    if (!block_bottom_shape(nx, ny, bc, &b)) return 0;
    const Sizes z(b, nx, ny, bc.type[0] == T_PERIODIC, bc.type[2] == T_PERIODIC);
    // the launches' items and the products' jobs: at most one and five a line and step
    return (z.keep + z.temp) * sizeof(double) + (size_t)2 * b.lines * (sizeof(int4) + 5 * sizeof(BlockMul));
}

cudaError_t launch_block_bottom(const BlockBottom& b, const DF& e, const DF& r, cudaStream_t st) {
    const unsigned rows = (b.m + kRowsPerCta - 1) / kRowsPerCta;
    cudaError_t err = cudaSuccess;
    for (int l = 0; l < b.steps && err == cudaSuccess; ++l)
        err = launch_step(k_bb_down, dim3(rows, b.ndown[l]), st, b, r, (int)(l == 0), b.items + b.odown[l]);
    for (int l = b.steps; l >= 0 && err == cudaSuccess; --l)
        err = launch_step(k_bb_up, dim3(rows, b.nup[l]), st, b, e, r, (int)(l == 0), b.items + b.oup[l]);
    return err;
}

int block_bottom_blocks(const BlockBottom& b, int l, bool up) {
    const int rows = (b.m + kRowsPerCta - 1) / kRowsPerCta;
    return up ? (l <= b.steps ? rows * b.nup[l] : 0) : (l < b.steps ? rows * b.ndown[l] : 0);
}

cudaError_t launch_block_jobs(const BlockJob* jobs, const int* pre, int njobs, int nblocks, int l, bool up,
                              cudaStream_t st) {
    if (njobs < 1 || nblocks < 1) return cudaSuccess;
    return up ? launch_step(k_bb_jobs<true>, dim3(nblocks), st, jobs, pre, njobs, l)
              : launch_step(k_bb_jobs<false>, dim3(nblocks), st, jobs, pre, njobs, l);
}

cudaError_t block_bottom_build(BlockBottom* b, const Geo& g, const BCd& bc, int nx, int ny, const BlockAlloc& mem,
                               cudaStream_t st, bool* ok) {
    *ok = false;
    const int m = b->m, B = b->lines;
    const size_t mm = (size_t)m * m;
    const bool px = bc.type[0] == T_PERIODIC, py = bc.type[2] == T_PERIODIC;
    const Sizes sz(*b, nx, ny, px, py);
    std::vector<Step> steps = elimination(B);
    if ((int)steps.size() > kBlockStepsMax) return cudaSuccess;
    Step top;
    top.up.push_back(int4{steps.back().down[0].x, -1, -1, 0});   // the line that is left
    steps.push_back(top);
    b->steps = (int)steps.size() - 1;
    std::vector<int4> items;
    for (int l = 0; l <= b->steps; ++l) {
        b->odown[l] = (int)items.size();
        b->ndown[l] = (int)steps[l].down.size();
        items.insert(items.end(), steps[l].down.begin(), steps[l].down.end());
        b->oup[l] = (int)items.size();
        b->nup[l] = (int)steps[l].up.size();
        items.insert(items.end(), steps[l].up.begin(), steps[l].up.end());
    }
    const int nc = sz.nc, nl = sz.nl, np = sz.np;
    const size_t ld = sz.ld, field = sz.field;
    double* keep = (double*)mem.get(mem.ctx, sz.keep * sizeof(double));
    b->mem = keep;
    b->items = (int4*)mem.get(mem.ctx, items.size() * sizeof(int4));
    double* temp = (double*)mem.get(mem.ctx, sz.temp * sizeof(double));
    std::vector<BlockMul> jobs;
    std::vector<int> n1, n2;
    double *D = keep, *P = keep + B * mm, *Q = keep + 2 * B * mm, *FG = keep + 3 * B * mm;
    double *A = temp, *C = temp + B * mm, *e0 = temp + 2 * B * mm, *e1 = e0 + mm, *out = e1 + mm;
    for (int l = 0; l < b->steps; ++l) {
        Step& s = steps[l];
        for (const int4& k : s.up) {
            if (k.y >= 0) s.first.push_back(BlockMul{P + k.x * mm, nullptr, D + k.x * mm, A + k.x * mm, nullptr, nullptr, 1.0});
            if (k.z >= 0) s.first.push_back(BlockMul{Q + k.x * mm, nullptr, D + k.x * mm, C + k.x * mm, nullptr, nullptr, 1.0});
        }
        for (const int4& k : s.down) {
            double *F = FG + k.w * mm, *G = F + mm;
            const int ln = k.y, rn = k.z;
            if (ln >= 0) s.first.push_back(BlockMul{F, nullptr, A + k.x * mm, D + ln * mm, nullptr, nullptr, 1.0});
            if (rn >= 0) s.first.push_back(BlockMul{G, nullptr, C + k.x * mm, D + rn * mm, nullptr, nullptr, 1.0});
            if (ln >= 0 || rn >= 0)
                s.second.push_back(BlockMul{D + k.x * mm, D + k.x * mm, ln >= 0 ? F : nullptr, C + (ln >= 0 ? ln : 0) * mm,
                                            rn >= 0 ? G : nullptr, A + (rn >= 0 ? rn : 0) * mm, -1.0});
            // a gone neighbour's other side becomes this line's neighbour
            if (ln >= 0)
                s.second.push_back(BlockMul{A + k.x * mm, (l == 0 && k.x == B - 1) ? e1 : nullptr, F, A + ln * mm, nullptr,
                                            nullptr, -1.0});
            if (rn >= 0)
                s.second.push_back(BlockMul{C + k.x * mm, (l == 0 && k.x == 0) ? e0 : nullptr, G, C + rn * mm, nullptr,
                                            nullptr, -1.0});
        }
        jobs.insert(jobs.end(), s.first.begin(), s.first.end());
        jobs.insert(jobs.end(), s.second.begin(), s.second.end());
        n1.push_back((int)s.first.size());
        n2.push_back((int)s.second.size());
    }
    BlockMul* djobs = (BlockMul*)mem.get(mem.ctx, jobs.size() * sizeof(BlockMul));
    int* fail = (int*)mem.get(mem.ctx, sizeof(int));
    cudaError_t err = cudaSuccess;
    int failed = 1;
    const auto step = [&](cudaError_t x) {
        if (err == cudaSuccess) err = x;
        return err == cudaSuccess;
    };
    if (keep && b->items && temp && djobs && fail) {
        b->dinv = D;
        b->p = P;
        b->q = Q;
        b->fg = FG;
        b->r = keep + (size_t)(3 * B + sz.nfg) * mm;
        b->bytes = sz.keep * sizeof(double) + items.size() * sizeof(int4);
        step(cudaMemsetAsync(fail, 0, sizeof(int), st));
        step(cudaMemsetAsync(keep, 0, sz.keep * sizeof(double), st));
        step(cudaMemsetAsync(temp, 0, sz.temp * sizeof(double), st));
        step(cudaMemcpyAsync(b->items, items.data(), items.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
        step(cudaMemcpyAsync(djobs, jobs.data(), jobs.size() * sizeof(BlockMul), cudaMemcpyHostToDevice, st));
        const auto at = [&](int k) { return DF{out + field * k + ld + 1, (int)ld}; };
        const DF phi = at(np), rhs = at(np + 1), res = at(np + 2);
        const dim3 blk(32, 8), gg((nx + 33) / 32, (ny + 9) / 8), gv((nx + 31) / 32, (ny + 7) / 8);
        for (int k = 0; k < np && err == cudaSuccess; ++k) {
            const int qc = k % nc, ql = k / nc;
            k_bb_probe<<<gg, blk, 0, st>>>(phi, nx, ny, px, py, b->along_y ? qc : ql, b->along_y ? ql : qc);
            step(cudaGetLastError());
            step(launch_fill(phi, g, bc, 1, 0, nx, ny, st));
            step(launch_apply(at(k), phi, rhs, g, bc, 1, nx, ny, 0, 0, st));
        }
        if (err == cudaSuccess) {
            k_bb_gather<<<B, 256, 0, st>>>(out, field, (int)ld, b->along_y, m, B, sz.pc, nc, nl, D, A, C, e0, e1);
            step(cudaGetLastError());
        }
        const size_t smem = (size_t)m * (m | 1) * sizeof(double);
        step(cudaFuncSetAttribute(k_bb_invert, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kBlockLineMax * (kBlockLineMax | 1) * sizeof(double))));
        const int tiles = (m + 31) / 32;
        size_t jo = 0;
        for (int l = 0; l <= b->steps && err == cudaSuccess; ++l) {
            k_bb_invert<<<b->nup[l], kInvThreads, smem, st>>>(D, b->items + b->oup[l], m, fail);
            step(cudaGetLastError());
            if (l == b->steps) break;
            k_bb_mul<<<dim3(tiles * tiles, n1[l]), 256, 0, st>>>(djobs + jo, m);
            k_bb_mul<<<dim3(tiles * tiles, n2[l]), 256, 0, st>>>(djobs + jo + n1[l], m);
            step(cudaGetLastError());
            jo += n1[l] + n2[l];
        }
        count_launch(np + 1 + 3 * b->steps + 1 + 2);
        if (err == cudaSuccess) {
            k_bb_rhs<<<gv, blk, 0, st>>>(rhs, nx, ny);
            step(cudaMemsetAsync(out + field * np, 0, field * sizeof(double), st));
            step(launch_block_bottom(*b, phi, rhs, st));
            step(launch_fill(phi, g, bc, 1, 0, nx, ny, st));
            step(launch_apply(res, phi, rhs, g, bc, 1, nx, ny, 1, 0, st));
        }
        if (err == cudaSuccess) {
            k_bb_check<<<1, 1024, 0, st>>>(res, nx, ny, fail);
            step(cudaGetLastError());
        }
        step(cudaMemcpyAsync(&failed, fail, sizeof(int), cudaMemcpyDeviceToHost, st));
        step(cudaStreamSynchronize(st));
    }
    for (void* p : {(void*)temp, (void*)djobs, (void*)fail}) mem.put(mem.ctx, p);
    *ok = err == cudaSuccess && !failed;
    if (!*ok) {
        for (void* p : {(void*)b->mem, (void*)b->items}) mem.put(mem.ctx, p);
        *b = BlockBottom{};
    }
    return err;
}

}  // namespace mgp
