// k_pcg.cu -- pressure projection: matrix-free preconditioned conjugate
// gradients on the MAC grid (replaces BridsonSolverGrid::solveIncompressibility,
// bridsonSolverGrid.cpp:244-293).
//
// System.  The reference assembles A with scale = dt/(rho h^2): diagonal =
// scale * (number of non-SOLID neighbours), off-diagonal = -scale towards fluid
// neighbours (calculateAMatrix, :40-77), and b = -(1/h) div(v2) [+ density
// term] (calculateRHS, :79-89).  Here the solver works on A' = A / scale, an
// integer 7-point stencil read straight from a 16-bit code per cell (fluid-
// neighbour mask + non-solid count), and b' = b / scale; the solution is the
// same p.  No matrix is stored.
//
// Preconditioner.  Incomplete Cholesky in red-black order (red = x+y+z even).
// Red rows have no earlier neighbours, so their pivots are the diagonal; a
// black pivot is d_B = ns_B - sum_j (1 + tau (nf_j - 1)) / ns_j over its red
// fluid neighbours j (the modified-IC fill compensation of the reference's
// MIC(0), tau = 0.97, with its safeguard d < 0.25 ns -> d = ns).  Applying M^-1
// is two half sweeps: z_B = (r_B + sum_j r_j / ns_j) / d_B, then
// z_R = (r_R + sum_k z_k) / ns_R; both colours are fully parallel.
//
// Precision (FSIM_PREC_MIXED).  Krylov vectors, stencil and preconditioner in
// FP32; dot products, alpha/beta and the convergence test in FP64; the
// solution accumulates in FP32 and is folded into an FP64 solution with the
// true residual b' - A' p recomputed in FP64 whenever the recursive residual
// has dropped by 1000x since the last fold ("reliable updates", refine_digits), and always
// before convergence is declared.  FSIM_PREC_FP32 never folds until the end;
// FSIM_PREC_FP64 runs every vector in FP64.
//
// Work layout.  Cells are grouped in 2x4x32 bricks (one 256-thread CTA pass
// per brick); only bricks holding a fluid cell are visited.  Per iteration
// three kernels: (1) s = z + beta s, q = A' s, s.q; (2) x += alpha s,
// r -= alpha q, black half-sweep, r.r / max|r|; (3) red half-sweep, z.r.
// Each reduction finishes in the last CTA to arrive (fixed order, so results
// are deterministic), which also updates the scalars in device memory; the
// host only polls a small state block every few iterations.
#include <algorithm>
#include <cmath>

#include "fsim_ctx.h"
#include "fsim_net.h"

#include <utility>

namespace {

template <typename... KArgs, typename... Args>
void launch_pdl(void (*kern)(KArgs...), unsigned grid, unsigned block, cudaStream_t st, Args&&... args) {
    launch_dep(kern, grid, block, 0, st, std::forward<Args>(args)...);
}

constexpr int BRX = 2, BRY = 4, BRZ = 32;
constexpr int PCG_THREADS = 256;
constexpr float TAU = 0.97f;
constexpr float SAFE = 0.25f;

// code bits
constexpr uint16_t CODE_FLUID = 0x8000;
__device__ __forceinline__ int code_ns(uint16_t c) { return (c >> 8) & 7; }
__device__ __forceinline__ int code_nf(uint16_t c) { return __popc(c & 0x3F); }

struct BrickGeo {
    GridGeom g;
    int nbx, nby, nbz;
    long long sx, sy;  // strides of +x and +y (+z is 1)
};

// neighbour offset k: +x, -x, +y, -y, +z, -z (bit k of the fluid mask)
__device__ __forceinline__ long long nb_off(const BrickGeo& B, int k) {
    const long long st = (k >> 1) == 0 ? B.sx : ((k >> 1) == 1 ? B.sy : 1ll);
    return (k & 1) ? -st : st;
}

// cell t of active brick bb = {bx, by, bz, b} (the compacted list's coordinates)
__device__ __forceinline__ bool brick_cell(const BrickGeo& B, int4 bb, int t, int& x, int& y, int& z,
                                           long long& c) {
    x = bb.x * BRX + t / (BRY * BRZ);
    y = bb.y * BRY + (t / BRZ) % BRY;
    z = bb.z * BRZ + t % BRZ;
    if (x >= B.g.nx || y >= B.g.ny || z >= B.g.nz) return false;
    c = gidx(B.g, x, y, z);
    return true;
}

__constant__ float c_fill[7][7];  // (1 + tau (nf - 1)) / ns
__constant__ float c_rcp[7];      // 1 / ns (1 for ns = 0)
__constant__ double c_nsd[7] = {0.0, 1.0, 2.0, 3.0, 4.0, 5.0, 6.0};

// Per-thread sums.  GB300 runs FP64 at a small fraction of its FP32 rate, so
// per-cell terms are summed in FP32 with compensation (Kahan), and only the
// per-thread totals enter the FP64 block / grid reduction.
template <typename T>
struct Acc {
    T s = 0;
    __device__ __forceinline__ void add(T x) { s += x; }
    __device__ __forceinline__ double value() const { return (double)s; }
};
template <>
struct Acc<float> {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};
template <typename T>
__device__ __forceinline__ T recip_ns(int ns);
template <>
__device__ __forceinline__ float recip_ns<float>(int ns) { return c_rcp[ns]; }
template <>
__device__ __forceinline__ double recip_ns<double>(int ns) { return ns > 0 ? 1.0 / ns : 1.0; }

__device__ __forceinline__ float black_pivot_inv(const uint16_t* code, long long c, uint16_t cc,
                                                 const BrickGeo& B) {
    const int ns = code_ns(cc);
    if (ns == 0) return 1.f;
    float d = (float)ns;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        if ((cc >> k) & 1) {
            const uint16_t cj = code[c + nb_off(B, k)];
            d -= c_fill[code_nf(cj)][code_ns(cj)];
        }
    }
    if (d < SAFE * ns) d = (float)ns;
    return __frcp_rn(d);
}

// ---- setup: codes, rhs, initial guess, brick activity ----------------------
struct SetupArgs {
    BrickGeo B;
    const uint8_t* flags;
    const float* v2[3];
    const float* avg;
    const float* guess;   // padded layout, or null
    const double* rhs_override;  // padded layout in A' units, or null
    int warm;             // FSIM_WARM_*
    int pressure_enabled;
    double avg_pressure, pressure_k;
    double inv_h, inv_scale;
    uint16_t* code;
    double* b;
    double* phi;
    uint8_t* brick_flag;
};

__global__ void k_setup(const SetupArgs a) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const GridGeom& g = a.B.g;
    if (c >= g.ncell) return;
    int x, y, z;
    cell_xyz(g, c, x, y, z);
    if (z >= g.nz) return;
    const uint8_t f = a.flags[c];
    if (f != C_WATER || x == 0 || y == 0 || z == 0 || x == g.nx - 1 || y == g.ny - 1 || z == g.nz - 1) {
        a.code[c] = 0;
        if (a.phi[c] != 0.0) a.phi[c] = 0.0;
        return;
    }
    uint16_t code = CODE_FLUID;
    int ns = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const uint8_t fn = a.flags[c + nb_off(a.B, k)];
        if (fn == C_WATER) code |= (uint16_t)(1u << k);
        if (fn != C_SOLID) ns++;
    }
    code |= (uint16_t)(ns << 8);
    a.code[c] = code;
    double bb;
    if (a.rhs_override) {
        bb = a.rhs_override[c];
    } else {
        const double sum = (double)a.v2[0][c] + (double)a.v2[1][c] + (double)a.v2[2][c] -
                           (double)a.v2[0][c - a.B.sx] - (double)a.v2[1][c - a.B.sy] -
                           (double)a.v2[2][c - 1];
        double rhs = -a.inv_h * sum;
        if (a.pressure_enabled) rhs += ((double)a.avg[c] - a.avg_pressure) * a.pressure_k;
        bb = rhs * a.inv_scale;
    }
    a.b[c] = bb;
    if (a.warm == FSIM_WARM_ZERO) a.phi[c] = 0.0;
    else if (a.warm == FSIM_WARM_GUESS && a.guess) a.phi[c] = (double)a.guess[c];
    const int bz = z / BRZ, by = y / BRY, bx = x / BRX;
    a.brick_flag[((long long)bx * a.B.nby + by) * a.B.nbz + bz] = 1;
}

// ordered compaction of active bricks (one CTA; 16 flags per thread and pass: 65,536
// bricks at 256^3 take 4 passes, 79 -> 8 us)
// each entry holds the brick's coordinates and index, int4 {bx, by, bz, b}, so
// the kernels over active bricks take them with one load, not three divisions
constexpr int COMPACT_THREADS = 1024, COMPACT_ITEMS = 16;
__global__ void __launch_bounds__(COMPACT_THREADS) k_compact_bricks(const uint8_t* flag, long long nb, int nby, int nbz,
                                                                    int4* xyz, int* count) {
    __shared__ int warp_tot[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (long long base = 0; base < nb; base += COMPACT_THREADS * COMPACT_ITEMS) {
        const long long j0 = base + (long long)threadIdx.x * COMPACT_ITEMS;
        // (the flags' allocation is 256-byte aligned; the tail is read byte by byte)
        alignas(16) uint8_t f[COMPACT_ITEMS];
        if (j0 + COMPACT_ITEMS <= nb) {
            *reinterpret_cast<uint4*>(f) = *reinterpret_cast<const uint4*>(flag + j0);
        } else {
            for (int k = 0; k < COMPACT_ITEMS; k++) f[k] = j0 + k < nb ? flag[j0 + k] : 0;
        }
        int mine = 0;
#pragma unroll
        for (int k = 0; k < COMPACT_ITEMS; k++) mine += f[k] != 0;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        int wt = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, wt, o);
            if (lane >= o) wt += t;
        }
        const int before = __shfl_sync(0xffffffffu, wt, warp > 0 ? warp - 1 : 0);
        int pos = carry + incl - mine + (warp > 0 ? before : 0);
        carry += __shfl_sync(0xffffffffu, wt, 31);
#pragma unroll
        for (int k = 0; k < COMPACT_ITEMS; k++)
            if (f[k]) {
                const unsigned ju = (unsigned)(j0 + k), t = ju / (unsigned)nbz, u = t / (unsigned)nby;
                xyz[pos++] = make_int4((int)u, (int)(t - u * (unsigned)nby), (int)(ju - t * (unsigned)nbz), (int)ju);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = carry;
}

struct PcgArgs {
    BrickGeo B;
    const int4* bxyz;  // active bricks, ascending: {bx, by, bz, b}
    const int* nactive;
    const uint16_t* code;
    const double* b;
    double* phi;
    PcgState* st;
    double* partials;
    unsigned* counter;
    double tol_abs, tol_rel;  // tolerance in A' units (abs) / relative
    double skip_bb;           // early-out threshold on b'.b' (reference: sum b^2 < 1e-7)
    int phi_zero;             // the solve starts from phi = 0 (its first residual is b)
};

template <typename T>
struct Vecs {
    T* r[2];
    T* s[2];
    T* z;
    T* q;
    T* x;  // accumulated solution (float plo for FP32/MIXED, double phi for FP64)
};

// r = b' - A' phi (FP64), store into r[rc]; reset x (FP32 accumulator) to 0.
// first = 1: also reduce |b'| and decide the reference's early-out.  FP64 arithmetic
// bounds this kernel (1/64 of the FP32 rate): the max norm comes from the stored
// residual, the rhs norm is needed by the first residual only, and a solve that
// starts from phi = 0 has r = b, one product per cell.
template <typename T>
__global__ void __launch_bounds__(PCG_THREADS) k_residual(const PcgArgs a, Vecs<T> v, int first, int reset_x) {
    __shared__ double scratch[PCG_THREADS * 3];
    T* r = (a.st->bufsel & 1) ? v.r[1] : v.r[0];
    double acc[3] = {0.0, -1e300, 0.0};  // rr, rmax, bb
    T rmaxT = (T)0;
    const bool from_zero = first && a.phi_zero;
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        const double bc = a.b[c];
        double rv = bc;
        if (!from_zero) {
            const double* phi = a.phi;
            rv = fma(-c_nsd[code_ns(cc)], phi[c], bc);
#pragma unroll
            for (int k = 0; k < 6; k++)
                if ((cc >> k) & 1) rv += phi[c + nb_off(a.B, k)];
            acc[0] += rv * rv;
        }
        const T rt = (T)rv;
        r[c] = rt;
        if (reset_x && sizeof(T) == 4) v.x[c] = (T)0;
        rmaxT = fmax(rmaxT, fabs(rt));
        if (first) acc[2] += bc * bc;
    }
    acc[1] = fmax(acc[1], (double)rmaxT);
    if (from_zero) acc[0] = acc[2];
    if (last_block_reduce<3>(acc, 0x2, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* s = a.st;
            s->rr = acc[0];
            s->rmax = acc[1];
            s->rr_update = acc[0];
            if (first) {
                s->bb = acc[2];
                s->tol_rel2 = a.tol_rel * a.tol_rel * acc[2];
                s->skip = acc[2] < a.skip_bb ? 1 : 0;
            }
            const bool conv = (s->tol_mode == FSIM_TOL_ABS_MAX) ? (acc[1] < s->tol_abs) : (acc[0] <= s->tol_rel2);
            s->converged = conv ? 1 : 0;
            s->done = (conv || s->skip) ? 1 : 0;
        }
    }
}

// black half-sweep from r[rc] (setup / after a fold)
template <typename T>
__global__ void __launch_bounds__(PCG_THREADS) k_black(const PcgArgs a, Vecs<T> v) {
    if (a.st->done) return;
    const int rc = a.st->bufsel & 1;
    const T* r = rc ? v.r[1] : v.r[0];
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        if (((x + y + z) & 1) == 0) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        T sum = r[c];
#pragma unroll
        for (int k = 0; k < 6; k++)
            if ((cc >> k) & 1) {
                const long long j = c + nb_off(a.B, k);
                sum += r[j] * recip_ns<T>(code_ns(a.code[j]));
            }
        v.z[c] = sum * (T)black_pivot_inv(a.code, c, cc, a.B);
    }
}

// red half-sweep + z.r over all fluid cells.
// mode 0: sigma = z.r, beta = 0 (setup)
// mode 1: beta = z.r / sigma, sigma_prev = sigma, sigma = z.r   (iteration)
// mode 2: beta = z.r / sigma_prev, sigma = z.r                  (after a fold)
template <typename T>
__global__ void __launch_bounds__(PCG_THREADS) k_red(const PcgArgs a, Vecs<T> v, int mode) {
    __shared__ double scratch[PCG_THREADS];
    if (a.st->done) return;
    const int rc = a.st->bufsel & 1;
    const T* r = rc ? v.r[1] : v.r[0];
    Acc<T> zr;
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        const T rv = r[c];
        T zv;
        if (((x + y + z) & 1) == 0) {
            T sum = rv;
#pragma unroll
            for (int k = 0; k < 6; k++)
                if ((cc >> k) & 1) sum += v.z[c + nb_off(a.B, k)];
            zv = sum * recip_ns<T>(code_ns(cc));
            v.z[c] = zv;
        } else {
            zv = v.z[c];
        }
        zr.add(zv * rv);
    }
    double acc[1] = {zr.value()};
    if (last_block_reduce<1>(acc, 0, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* s = a.st;
            const double sig = acc[0];
            if (mode == 0) {
                s->beta = 0.0;
                s->sigma = sig;
                s->sigma_prev = sig;
            } else if (mode == 1) {
                s->beta = sig / s->sigma;
                s->sigma_prev = s->sigma;
                s->sigma = sig;
            } else {
                s->beta = sig / s->sigma_prev;
                s->sigma = sig;
            }
            if (!isfinite(s->beta)) {
                s->nan = 1;
                s->done = 1;
            }
        }
    }
}

// s_new = z + beta s_old; q = A' s_new; alpha = sigma / (s.q)
template <typename T>
__global__ void __launch_bounds__(PCG_THREADS) k_spmv(const PcgArgs a, Vecs<T> v) {
    __shared__ double scratch[PCG_THREADS];
    if (a.st->done) return;
    const int sc = (a.st->bufsel >> 1) & 1;
    const double beta = a.st->beta;
    const T* so = sc ? v.s[1] : v.s[0];
    T* sn = sc ? v.s[0] : v.s[1];
    Acc<T> sq;
    const T betaT = (T)beta;
    const bool beta0 = beta == 0.0;
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        // beta = 0 (first iteration, after a restart): s = z exactly, without
        // reading s_old (which may hold a previous solve's non-finite values)
        const T snc = beta0 ? v.z[c] : v.z[c] + betaT * so[c];
        T qv = (T)code_ns(cc) * snc;
#pragma unroll
        for (int k = 0; k < 6; k++)
            if ((cc >> k) & 1) {
                const long long j = c + nb_off(a.B, k);
                qv -= beta0 ? v.z[j] : v.z[j] + betaT * so[j];
            }
        sn[c] = snc;
        v.q[c] = qv;
        sq.add(snc * qv);
    }
    double acc[1] = {sq.value()};
    if (last_block_reduce<1>(acc, 0, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* s = a.st;
            s->alpha = s->sigma / acc[0];
            if (!isfinite(s->alpha)) {
                s->nan = 1;
                s->done = 1;
            }
            s->bufsel ^= 2;  // s buffers swap
        }
    }
}

// x += alpha s; r_new = r - alpha q; r.r, max|r|; then on r_new the black half of the
// red-black IC solve (the red half is k_red)
template <typename T>
__global__ void __launch_bounds__(PCG_THREADS) k_update(const PcgArgs a, Vecs<T> v) {
    __shared__ double scratch[PCG_THREADS * 2];
    if (a.st->done) return;
    const int rc = a.st->bufsel & 1, sc = (a.st->bufsel >> 1) & 1;
    const T alpha = (T)a.st->alpha;
    const T* ro = rc ? v.r[1] : v.r[0];
    T* rn = rc ? v.r[0] : v.r[1];
    const T* s = sc ? v.s[1] : v.s[0];
    Acc<T> rr;
    T rmax = (T)0;
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        v.x[c] += alpha * s[c];
        const T rv = ro[c] - alpha * v.q[c];
        rn[c] = rv;
        rr.add(rv * rv);
        rmax = fmax(rmax, fabs(rv));
        if ((x + y + z) & 1) {
            T sum = rv;
#pragma unroll
            for (int k = 0; k < 6; k++)
                if ((cc >> k) & 1) {
                    const long long j = c + nb_off(a.B, k);
                    const uint16_t cj = a.code[j];
                    sum += (ro[j] - alpha * v.q[j]) * recip_ns<T>(code_ns(cj));
                }
            v.z[c] = sum * (T)black_pivot_inv(a.code, c, cc, a.B);
        }
    }
    double acc[2] = {rr.value(), (double)rmax};
    if (last_block_reduce<2>(acc, 0x2, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* st = a.st;
            st->rr = acc[0];
            st->rmax = acc[1];
            st->it += 1;
            st->bufsel ^= 1;  // r buffers swap
            const bool conv = (st->tol_mode == FSIM_TOL_ABS_MAX) ? (acc[1] < st->tol_abs) : (acc[0] <= st->tol_rel2);
            st->converged = conv ? 1 : 0;
            if (conv || st->it >= st->max_iters || !isfinite(acc[0])) st->done = 1;
            if (!isfinite(acc[0])) st->nan = 1;
            // the FP32 recursion is trusted for a fold_drop fall of r.r, then the
            // solution is folded into FP64 and the iteration restarts
            if (st->fold_enabled && acc[0] < st->fold_drop * st->rr_update) {
                st->need_fold = 1;
                st->done = 1;
            }
        }
    }
}

// ---- geometric multigrid preconditioner ------------------------------------
//
// z = M^-1 r by one V-cycle.  Level l + 1 halves every dimension (ceil); a
// coarse cell is fluid if any child is fluid, else air if any child is air,
// else solid.  Level 0 is the integer stencil; a coarse level's operator is a
// 7-point stencil built from the finer level's faces (k_mg_code).  In the fine
// level's units the level-l operator is L_l / 4^l, so the coarse right-hand
// side is 4 R (f - L x) with R = P^T / 8 and P the cell-centred trilinear
// prolongation (weights 3/4 and 1/4 per axis) divided by the weight of the
// coarse neighbours that are not solid (k_mg_pscale).  The smoother is
// red-black Gauss-Seidel, NU sweeps red->black before the coarse correction and
// black->red after it; the coarsest level (at most 4 cells per axis) is smoothed
// BOTTOM times each way inside one CTA.  Starting every level from zero, the
// V-cycle is a fixed symmetric linear operator, as CG requires.
//
// Both rules are what makes V(1,1) converge like the textbook cycle here:
// without the division interpolation loses a quarter of a constant at every
// wall, and with coarse cells rediscretised from their own kinds a cell cut by
// the free surface is tied to p = 0 as weakly as a full one.  Iterations to
// 1e-6 with one sweep on every level (128^3 dam break / porous random mask):
// 26 / 55 with neither, 16 / 11 with the face operator alone, 9 / 9 with both,
// the same from 32^3 to 256^3.  With the rediscretised operator the best sweep
// counts were 1-2 / 4 / 6 / 8, plus three band sweeps at the surface:
// 17 iterations and 12.1 ms at 256^3, against 8 iterations and 5.0 ms now
// (one GB300, half-filled box).
//
// MIXED precision: the FP32 recursion is folded into the FP64 solution (true
// FP64 residual, CG restart) each time the residual norm fell this many decades.
// The FP32 correction restarts from zero at every fold, so the drift between the
// recursive and the true residual stays near FP32 rounding of the fold's
// residual, far below a 10^-3 drop.  One decade per fold (the first setting)
// cost 5 refinements per 1e-6 solve at 256^3; four or five decades also need
// two, at the same time.
constexpr int MIXED_REFINE_DIGITS = 3;
// Sweeps per level: level 0 / separately launched coarse levels / cluster levels,
// ms of a solve to 1e-6 (32^3 and 128^3 dam break, 256^3 half filled, random
// mask 72x100x85): 1/1/1 0.73, 1.52, 5.05, 1.45; 1/2/2 0.68, 1.44, 4.95, 1.38;
// 2/2/2 0.70, 1.41, 5.28, 1.38; 2/1/1 0.76, 1.66, 5.90, 1.47.  Band sweeps no
// longer pay: 1/1/1 with two, 0.93, 1.76, 5.35, 1.84.
constexpr int MG_NU_DEFAULT = 1;         // level 0
constexpr int MG_NU_COARSE_DEFAULT = 2;  // all coarser levels
constexpr int MG_BOTTOM_SWEEPS = 4;  // on the <= 4^3 bottom level
constexpr int MG_BOTTOM_MAX = 4096;

struct MGLev {
    int nx, ny, nz, pz;
    const uint16_t* code;   // level 0
    const uint32_t* ccode;  // levels >= 1 (coarse_* helpers)
    float* x;
    const float* f;
    const float* f1;  // level 0: the rhs is the current PCG residual buffer (r[0] or r[1])
    float* r;
};

__device__ __forceinline__ const float* mg_rhs(const PcgArgs& A, const MGLev& L) {
    return (L.f1 && (A.st->bufsel & 1)) ? L.f1 : L.f;
}

// Coarse cell code (levels >= 1): bits 3k..3k+2 the open quarters (0..4) of the
// face towards neighbour k (+x, -x, +y, -y, +z, -z), bits 18-22 the Dirichlet
// weight in eighths, bits 23-28 the interpolation scale (below); 0 = no unknown.
constexpr uint32_t CC_OP = 0x7FFFFF;      // faces and Dirichlet weight
constexpr uint32_t CC_INTERIOR = 0x24924; // six open faces, no Dirichlet weight
constexpr int CC_DIRICHLET = 18, CC_SCALE = 23;
constexpr int DIRICHLET_MAX = 24;         // eighths
// marks of the copies in shared memory
constexpr uint32_t CS_ODD = 1u << 29, CS_HIGH = 1u << 30;  // odd x + y + z; upper cell of a z pair

// eight times the diagonal: two per open quarter face plus the Dirichlet eighths
__device__ __forceinline__ int coarse_diag8(uint32_t cc) {
    const uint32_t a = (cc & 0x71C7u) + ((cc >> 3) & 0x71C7u);
    return 2 * (int)((a + (a >> 6) + (a >> 12)) & 0x3Fu) + (int)((cc >> CC_DIRICHLET) & 31u);
}
// small unsigned integer to float without the quarter-rate conversion unit
__device__ __forceinline__ float small_float(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.f; }
__device__ __forceinline__ float coarse_face(uint32_t cc, int k) { return small_float((cc >> (3 * k)) & 7u); }
// f + neighbours over the diagonal; sum4 = sum of (quarters * neighbour value)
__device__ __forceinline__ float coarse_solve(uint32_t cc, float f, float sum4) {
    return __fdividef(8.f * f + 2.f * sum4, small_float((uint32_t)coarse_diag8(cc)));
}
__device__ __forceinline__ float coarse_resid(uint32_t cc, float f, float x, float sum4) {
    return f - (0.125f * small_float((uint32_t)coarse_diag8(cc)) * x - 0.25f * sum4);
}

// Interpolation scale.  The trilinear weights (27, 9, 9, 9, 3, 3, 3, 1)/64 of a
// cell's eight coarse neighbours are divided by the sum over those that are
// not solid (k / 64), so that interpolation reproduces constants next to walls
// (zero normal derivative) and still falls to zero towards air (p = 0).  Codes
// store 64 - k (0 in the interior; the cell's own parent is fluid, so k >= 27):
// level 0 in the code's six spare bits, coarse levels in bits 23-28.
__constant__ float c_pscale[64];  // 64 / (64 - i)
__device__ __forceinline__ float code_pscale(uint16_t c) { return c_pscale[((c >> 6) & 3) | ((c >> 9) & 0x3C)]; }
__device__ __forceinline__ float coarse_pscale(uint32_t c) { return c_pscale[(c >> CC_SCALE) & 63u]; }

// ---- quad kernels -----------------------------------------------------------
// Every multigrid kernel (and the MG-path PCG kernels) gives each thread a quad:
// four consecutive z cells of one row, 16-byte aligned (every level pads z to
// a multiple of 4).  The centre and the +-x / +-y neighbour quads are single
// float4 loads, the +-z neighbours come from the quad itself plus one scalar on
// either side, and the four cell codes are one 8-byte load.  Level 0 walks the
// active bricks (64 quads per 2x4x32 brick, four bricks per 256-thread pass);
// coarser levels walk all their quads.
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void unpack4(const float4 f, float (&v)[4]) {
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void codes4(const uint16_t* code, long long c0, uint16_t (&cc)[4]) {
    const uint2 w = *reinterpret_cast<const uint2*>(code + c0);
    cc[0] = (uint16_t)(w.x & 0xFFFFu);
    cc[1] = (uint16_t)(w.x >> 16);
    cc[2] = (uint16_t)(w.y & 0xFFFFu);
    cc[3] = (uint16_t)(w.y >> 16);
}
__device__ __forceinline__ bool any_fluid(const uint16_t (&cc)[4]) {
    return ((cc[0] | cc[1] | cc[2] | cc[3]) & CODE_FLUID) != 0;
}
__device__ __forceinline__ void codes4(const uint32_t* code, long long c0, uint32_t (&cc)[4]) {
    const uint4 w = *reinterpret_cast<const uint4*>(code + c0);
    cc[0] = w.x; cc[1] = w.y; cc[2] = w.z; cc[3] = w.w;
}
__device__ __forceinline__ bool any_fluid(const uint32_t (&cc)[4]) {
    return ((cc[0] | cc[1] | cc[2] | cc[3]) & CC_OP) != 0;
}
__device__ __forceinline__ bool is_fluid(uint16_t c) { return (c & CODE_FLUID) != 0; }
__device__ __forceinline__ bool is_fluid(uint32_t c) { return (c & CC_OP) != 0; }

// a field around a quad: centre and the four face-neighbour quads, plus z ends
struct Q7 {
    float c[4], xp[4], xm[4], yp[4], ym[4];
    float zm, zp;
};
// neighbour quads outside the level read as zero (their mask bits are clear)
__device__ __forceinline__ void load_q7(Q7& q, const float* v, long long c0, const MGLev& L, int x, int y, int z0) {
    const long long sx = (long long)L.pz * L.ny, sy = L.pz;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    unpack4(ld4(v + c0), q.c);
    unpack4(x + 1 < L.nx ? ld4(v + c0 + sx) : zero, q.xp);
    unpack4(x > 0 ? ld4(v + c0 - sx) : zero, q.xm);
    unpack4(y + 1 < L.ny ? ld4(v + c0 + sy) : zero, q.yp);
    unpack4(y > 0 ? ld4(v + c0 - sy) : zero, q.ym);
    q.zm = z0 > 0 ? v[c0 - 1] : 0.f;
    q.zp = z0 + 4 < L.pz ? v[c0 + 4] : 0.f;
}
__device__ __forceinline__ void codes4_nb(const uint16_t* code, long long c0, bool ok, uint16_t (&cc)[4]) {
    if (ok) codes4(code, c0, cc);
    else cc[0] = cc[1] = cc[2] = cc[3] = 0;
}
// sum over the fluid neighbours (mask bits of cc) of lane i
__device__ __forceinline__ float nbsum(const Q7& q, int i, uint16_t cc) {
    float s = 0.f;
    if (cc & 1) s += q.xp[i];
    if (cc & 2) s += q.xm[i];
    if (cc & 4) s += q.yp[i];
    if (cc & 8) s += q.ym[i];
    if (cc & 16) s += (i < 3) ? q.c[i + 1] : q.zp;
    if (cc & 32) s += (i > 0) ? q.c[i - 1] : q.zm;
    return s;
}

// the same on a coarse level: sum of (open quarters * neighbour value)
__device__ __forceinline__ float nbsum4(const Q7& q, int i, uint32_t cc) {
    const float zp = (i < 3) ? q.c[i + 1] : q.zp, zm = (i > 0) ? q.c[i - 1] : q.zm;
    if ((cc & CC_OP) == CC_INTERIOR) return 4.f * (q.xp[i] + q.xm[i] + q.yp[i] + q.ym[i] + zp + zm);
    // closed faces are skipped, not multiplied by zero: a cell without an unknown
    // may hold an earlier solve's non-finite value
    float s = 0.f;
    if (cc & 7u) s += coarse_face(cc, 0) * q.xp[i];
    if (cc & (7u << 3)) s += coarse_face(cc, 1) * q.xm[i];
    if (cc & (7u << 6)) s += coarse_face(cc, 2) * q.yp[i];
    if (cc & (7u << 9)) s += coarse_face(cc, 3) * q.ym[i];
    if (cc & (7u << 12)) s += coarse_face(cc, 4) * zp;
    if (cc & (7u << 15)) s += coarse_face(cc, 5) * zm;
    return s;
}

// Gauss-Seidel value and residual of lane i, on either kind of level
__device__ __forceinline__ float gs_value(const Q7& q, int i, uint16_t cc, float f, bool first) {
    return (first ? f : f + nbsum(q, i, cc)) * c_rcp[code_ns(cc)];
}
__device__ __forceinline__ float gs_value(const Q7& q, int i, uint32_t cc, float f, bool first) {
    return coarse_solve(cc, f, first ? 0.f : nbsum4(q, i, cc));
}
__device__ __forceinline__ float resid_value(const Q7& q, int i, uint16_t cc, float f) {
    return f - ((float)code_ns(cc) * q.c[i] - nbsum(q, i, cc));
}
__device__ __forceinline__ float resid_value(const Q7& q, int i, uint32_t cc, float f) {
    return coarse_resid(cc, f, q.c[i], nbsum4(q, i, cc));
}
__device__ __forceinline__ float pscale_of(uint16_t c) { return code_pscale(c); }
__device__ __forceinline__ float pscale_of(uint32_t c) { return coarse_pscale(c); }
template <bool FINE>
struct LevCode { using T = uint16_t; static __device__ __forceinline__ const T* of(const MGLev& L) { return L.code; } };
template <>
struct LevCode<false> { using T = uint32_t; static __device__ __forceinline__ const T* of(const MGLev& L) { return L.ccode; } };

// all quads of a coarse level, thread i0 + k * step
// (x, y, z0) of quad i of a level, in 32-bit arithmetic (levels stay below 2^31 cells)
__device__ __forceinline__ void quad_xyz(const MGLev& L, long long i, int& x, int& y, int& z0) {
    const unsigned iu = (unsigned)i, qz = (unsigned)(L.pz >> 2), ny = (unsigned)L.ny;
    const unsigned t = iu / qz;
    z0 = (int)(iu - t * qz) << 2;
    const unsigned u = t / ny;
    y = (int)(t - u * ny);
    x = (int)u;
}

template <typename F>
__device__ __forceinline__ void mg_for_range(const MGLev& L, long long i0, long long step, F&& fn) {
    const long long n = (long long)L.nx * L.ny * (L.pz >> 2);
    for (long long i = i0; i < n; i += step) {
        int x, y, z0;
        quad_xyz(L, i, x, y, z0);
        fn(x, y, z0, ((long long)x * L.ny + y) * L.pz + z0);
    }
}

template <bool FINE, typename F>
__device__ __forceinline__ void mg_for_quads(const PcgArgs& A, const MGLev& L, F&& fn) {
    if (FINE) {
        const int nact = *A.nactive;
        const int sub = threadIdx.x >> 6, q = threadIdx.x & 63;
        for (int bk = blockIdx.x * 4 + sub; bk < nact; bk += gridDim.x * 4) {
            const int4 bb = A.bxyz[bk];
            const int x = bb.x * BRX + (q >> 5), y = bb.y * BRY + ((q >> 3) & 3), z0 = bb.z * BRZ + ((q & 7) << 2);
            if (x >= L.nx || y >= L.ny || z0 >= L.nz) continue;
            fn(x, y, z0, ((long long)x * L.ny + y) * L.pz + z0);
        }
    } else {
        mg_for_range(L, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x, fn);
    }
}

__device__ __forceinline__ long long lev_sx(const MGLev& L) { return (long long)L.pz * L.ny; }

// one red-black Gauss-Seidel half sweep of a quad; first: the other colour is still zero
template <bool FINE>
__device__ __forceinline__ void smooth_quad(const MGLev& L, const float* rhs, int color, int first, int x, int y,
                                            int z0, long long c0) {
    // every load is issued before the fluid test (one round trip, not two; the
    // levels sit in L2, so the loads of quads without fluid are cheap)
    typename LevCode<FINE>::T cc[4];
    codes4(LevCode<FINE>::of(L), c0, cc);
    float f[4];
    unpack4(ld4(rhs + c0), f);
    Q7 q;
    if (first) unpack4(ld4(L.x + c0), q.c);
    else load_q7(q, L.x, c0, L, x, y, z0);
    if (!any_fluid(cc)) return;
    const int par = (x + y + z0) & 1;
    float out[4] = {q.c[0], q.c[1], q.c[2], q.c[3]};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (((par ^ i) & 1) != color || !is_fluid(cc[i])) continue;
        out[i] = gs_value(q, i, cc[i], f[i], first != 0);
    }
    st4(L.x + c0, out);
}

template <bool FINE>
__global__ void __launch_bounds__(PCG_THREADS) k_mg_smooth(const PcgArgs A, MGLev L, int color, int first) {
    pdl_enter();
    if (A.st->done) return;
    const float* rhs = mg_rhs(A, L);
    mg_for_quads<FINE>(A, L, [&](int x, int y, int z0, long long c0) { smooth_quad<FINE>(L, rhs, color, first, x, y, z0, c0); });
}

// the last post-smoothing half sweep (red, level 0) fused with z.r (modes 0/1 as k_red)
__global__ void __launch_bounds__(PCG_THREADS) k_mg_smooth_dot(const PcgArgs A, MGLev L, int mode) {
    __shared__ double scratch[PCG_THREADS];
    pdl_enter();
    if (A.st->done) return;
    const float* rhs = mg_rhs(A, L);
    Acc<float> zr;
    mg_for_quads<true>(A, L, [&](int x, int y, int z0, long long c0) {
        uint16_t cc[4];
        codes4(L.code, c0, cc);
        if (!any_fluid(cc)) return;
        float f[4];
        unpack4(ld4(rhs + c0), f);
        Q7 q;
        load_q7(q, L.x, c0, L, x, y, z0);
        const int par = (x + y + z0) & 1;
        float out[4] = {q.c[0], q.c[1], q.c[2], q.c[3]};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (!(cc[i] & CODE_FLUID)) continue;
            if (((par ^ i) & 1) == 0) out[i] = (f[i] + nbsum(q, i, cc[i])) * c_rcp[code_ns(cc[i])];
            zr.add(out[i] * f[i]);
        }
        st4(L.x + c0, out);
    });
    double acc[1] = {zr.value()};
    if (last_block_reduce<1>(acc, 0, A.partials, A.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* s = A.st;
            const double sig = acc[0];
            if (mode == 0) {
                s->beta = 0.0;
                s->sigma = sig;
                s->sigma_prev = sig;
            } else {
                s->beta = sig / s->sigma;
                s->sigma_prev = s->sigma;
                s->sigma = sig;
            }
            if (!isfinite(s->beta)) {
                s->nan = 1;
                s->done = 1;
            }
        }
    }
}

// r = (f - A x) times the interpolation scale (restriction is the transpose of
// the scaled interpolation)
template <bool FINE>
__device__ __forceinline__ void residual_quad(const MGLev& L, const float* rhs, int x, int y, int z0, long long c0) {
    typename LevCode<FINE>::T cc[4];
    codes4(LevCode<FINE>::of(L), c0, cc);
    float f[4];
    unpack4(ld4(rhs + c0), f);
    Q7 q;
    load_q7(q, L.x, c0, L, x, y, z0);
    if (FINE && !any_fluid(cc)) return;  // (stays zero; a coarse level's quad is written below)
    float out[4];
#pragma unroll
    for (int i = 0; i < 4; i++) out[i] = is_fluid(cc[i]) ? resid_value(q, i, cc[i], f[i]) * pscale_of(cc[i]) : 0.f;
    st4(L.r + c0, out);
}

template <bool FINE>
__global__ void __launch_bounds__(PCG_THREADS) k_mg_residual(const PcgArgs A, MGLev L) {
    pdl_enter();
    if (A.st->done) return;
    const float* rhs = mg_rhs(A, L);
    mg_for_quads<FINE>(A, L, [&](int x, int y, int z0, long long c0) { residual_quad<FINE>(L, rhs, x, y, z0, c0); });
}

// coarse f = 0.5 * sum_fine P[f,C] r_f  (= 4 R r), per coarse quad: the fine
// plane 2 cx + dx's share (r is zero off the fluid: mg_setup clears level 0's, the
// coarser residual passes write every quad)
__device__ __forceinline__ void restrict_plane(const MGLev& F, int cx, int cy, int cz0, int dx, float (&sum)[4]) {
    const int fx = 2 * cx + dx;
    if (fx < 0 || fx >= F.nx) return;
    const float wx = (dx == 0 || dx == 1) ? 0.375f : 0.125f;
    const int fz = 2 * cz0;  // fine z fz - 1 .. fz + 8
#pragma unroll
    for (int dy = -1; dy <= 2; dy++) {
        const int fy = 2 * cy + dy;
        if (fy < 0 || fy >= F.ny) continue;
        const float wxy = wx * ((dy == 0 || dy == 1) ? 0.75f : 0.25f);
        const float* row = F.r + ((long long)fx * F.ny + fy) * F.pz + fz;
        float fr[10], v[4] = {0.f, 0.f, 0.f, 0.f}, w[4] = {0.f, 0.f, 0.f, 0.f};
        fr[0] = fz > 0 ? row[-1] : 0.f;
        if (fz < F.pz) unpack4(ld4(row), v);
        if (fz + 4 < F.pz) unpack4(ld4(row + 4), w);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            fr[1 + e] = v[e];
            fr[5 + e] = w[e];
        }
        fr[9] = fz + 8 < F.pz ? row[8] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++)
            sum[j] += wxy * (0.25f * fr[2 * j] + 0.75f * fr[1 + 2 * j] + 0.75f * fr[2 + 2 * j] + 0.25f * fr[3 + 2 * j]);
    }
}
__device__ __forceinline__ void restrict_quad(const MGLev& F, const MGLev& Cl, int cx, int cy, int cz0, long long ci) {
    uint32_t ccc[4];
    codes4(Cl.ccode, ci, ccc);
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    for (int dx = -1; dx <= 2; dx++) restrict_plane(F, cx, cy, cz0, dx, sum);
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (is_fluid(ccc[j])) const_cast<float*>(Cl.f)[ci + j] = sum[j];
}

// Four lanes (l, l + 8, l + 16, l + 24) share a coarse quad, one fine plane each, and
// a warp's eight quads are neighbours along z (full sectors): with one thread
// per quad (128 loads one after the other, fine codes among them) a pass took 9-10 us
// on a small level and 27 us from a half-filled 256^3, now 3-4 and 24.  The coarse
// level's first half sweep from zero (red: x = f / diagonal) needs nothing else and is
// done on the way.
__global__ void __launch_bounds__(PCG_THREADS) k_mg_restrict(const PcgState* st, MGLev F, MGLev Cl, int skip) {
    pdl_enter();
    if (st->done) return;
    const long long n = (long long)Cl.nx * Cl.ny * (Cl.pz >> 2);
    const int k = (threadIdx.x & 31) >> 3;
    const long long step = ((long long)gridDim.x * blockDim.x) >> 2;
    // whole warps leave together: eight quads per warp, the last ones clamped
    for (long long i0 = ((long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) >> 2; i0 < n; i0 += step) {
        const long long i = i0 + (threadIdx.x & 7);
        const bool in = i < n;
        int cx, cy, cz0;
        quad_xyz(Cl, in ? i : n - 1, cx, cy, cz0);
        const long long ci = ((long long)cx * Cl.ny + cy) * Cl.pz + cz0;
        const uint32_t cc = Cl.ccode[ci + k];
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        // quads without a fluid cell (half of a dam break's) read nothing: 31 to 23 us from
        // 256^3.  Not on small levels, where the wait for the codes costs 1 us of 4.
        const unsigned fluid = skip ? __ballot_sync(0xffffffffu, is_fluid(cc)) : 0xffffffffu;
        if ((fluid >> (threadIdx.x & 7)) & 0x01010101u) restrict_plane(F, cx, cy, cz0, k - 1, sum);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], 8);
            sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], 16);
        }
        if (in && is_fluid(cc)) {
            const float f = k == 0 ? sum[0] : k == 1 ? sum[1] : k == 2 ? sum[2] : sum[3];
            const_cast<float*>(Cl.f)[ci + k] = f;
            if (((cx + cy + cz0 + k) & 1) == 0) Cl.x[ci + k] = coarse_solve(cc, f, 0.f);
        }
    }
}

// fine x += P x_coarse on fluid fine cells, per fine quad: the quad's coarse z
// neighbours are z0/2 - 1 .. z0/2 + 2
template <bool FINE>
__device__ __forceinline__ void prolong_quad(const MGLev& F, const MGLev& Cl, int x, int y, int z0, long long c0) {
    typename LevCode<FINE>::T cc[4];
    codes4(LevCode<FINE>::of(F), c0, cc);
    if (!any_fluid(cc)) return;
    const int px = (x & 1) ? x >> 1 : (x >> 1) - 1;  // lower coarse neighbour per axis
    const int py = (y & 1) ? y >> 1 : (y >> 1) - 1;
    const float wlx = (x & 1) ? 0.75f : 0.25f, wly = (y & 1) ? 0.75f : 0.25f;
    const int zc = (z0 >> 1) - 1;
    // coarse z zc .. zc + 3: with h = z0 / 2 even, either the quad at h plus the
    // value below it (h = 0 mod 4) or the quad at h - 2 plus the value above it
    const int hq = (z0 >> 1) & ~3;
    const bool lowq = ((z0 >> 1) & 3) == 0;
    const int ze = lowq ? zc : hq + 4;  // the extra value's z
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int o = 0; o < 4; o++) {
        const int ox = o >> 1, oy = o & 1;
        const int cx = px + ox, cy = py + oy;
        if (cx < 0 || cy < 0 || cx >= Cl.nx || cy >= Cl.ny) continue;
        const float wxy = (ox ? 1.f - wlx : wlx) * (oy ? 1.f - wly : wly);
        const long long row = ((long long)cx * Cl.ny + cy) * Cl.pz;
        // (x is zero where the coarse cell is not fluid: k_mg_code)
        float qv[4];
        unpack4(ld4(Cl.x + row + hq), qv);
        const float ev = ze >= 0 && ze < Cl.pz ? Cl.x[row + ze] : 0.f;
        float cv[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            // lowq: zc = hq - 1 (the extra value), then hq .. hq + 2; else hq + 1 .. hq + 3, then hq + 4
            cv[k] = lowq ? (k == 0 ? ev : qv[k - 1]) : (k == 3 ? ev : qv[k + 1]);
        // lanes: z0 (lower zc, w 1/4), z0+1 (zc+1, 3/4), z0+2 (zc+1, 1/4), z0+3 (zc+2, 3/4)
        sum[0] += wxy * (0.25f * cv[0] + 0.75f * cv[1]);
        sum[1] += wxy * (0.75f * cv[1] + 0.25f * cv[2]);
        sum[2] += wxy * (0.25f * cv[1] + 0.75f * cv[2]);
        sum[3] += wxy * (0.75f * cv[2] + 0.25f * cv[3]);
    }
    float xv[4];
    unpack4(ld4(F.x + c0), xv);
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (is_fluid(cc[i])) xv[i] += sum[i] * pscale_of(cc[i]);
    st4(F.x + c0, xv);
}

template <bool FINE>
__global__ void __launch_bounds__(PCG_THREADS) k_mg_prolong(const PcgArgs A, MGLev F, MGLev Cl) {
    pdl_enter();
    if (A.st->done) return;
    mg_for_quads<FINE>(A, F, [&](int x, int y, int z0, long long c0) { prolong_quad<FINE>(F, Cl, x, y, z0, c0); });
}

// ---- free-surface band of the finest level ------------------------------------
// Quads with a fluid cell whose cells or six neighbouring cells include an
// interface cell (fluid with an air neighbour: fewer fluid than non-solid
// neighbours).  Extra red-black sweeps on this band only (mg_boundary_sweeps)
// target the error the coarse-grid correction leaves at the free surface,
// where the coarse levels represent the Dirichlet boundary worst.
__device__ __forceinline__ bool iface_cell(uint16_t c) { return (c & CODE_FLUID) && code_ns(c) != code_nf(c); }

__global__ void __launch_bounds__(PCG_THREADS) k_bnd_list(const PcgArgs A, MGLev L, int4* out, int* count) {
    const long long sx = lev_sx(L), sy = L.pz;
    mg_for_quads<true>(A, L, [&](int x, int y, int z0, long long c0) {
        uint16_t cc[4];
        codes4(L.code, c0, cc);
        if (!any_fluid(cc)) return;
        bool in = false;
        uint16_t nb[4];
#pragma unroll
        for (int i = 0; i < 4; i++) in |= iface_cell(cc[i]);
        codes4_nb(L.code, c0 + sx, x + 1 < L.nx, nb);
#pragma unroll
        for (int i = 0; i < 4; i++) in |= iface_cell(nb[i]);
        codes4_nb(L.code, c0 - sx, x > 0, nb);
#pragma unroll
        for (int i = 0; i < 4; i++) in |= iface_cell(nb[i]);
        codes4_nb(L.code, c0 + sy, y + 1 < L.ny, nb);
#pragma unroll
        for (int i = 0; i < 4; i++) in |= iface_cell(nb[i]);
        codes4_nb(L.code, c0 - sy, y > 0, nb);
#pragma unroll
        for (int i = 0; i < 4; i++) in |= iface_cell(nb[i]);
        if (z0 > 0) in |= iface_cell(L.code[c0 - 1]);
        if (z0 + 4 < L.pz) in |= iface_cell(L.code[c0 + 4]);
        if (in) out[atomicAdd(count, 1)] = make_int4(x, y, z0, 0);
    });
}

// one red-black half sweep over the band's quads
__global__ void __launch_bounds__(PCG_THREADS) k_mg_smooth_bnd(const PcgArgs A, MGLev L, const int4* list,
                                                               const int* count, int color) {
    pdl_enter();
    if (A.st->done) return;
    const float* rhs = mg_rhs(A, L);
    const int n = *count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 q = list[i];
        smooth_quad<true>(L, rhs, color, 0, q.x, q.y, q.z, ((long long)q.x * L.ny + q.y) * L.pz + q.z);
    }
}

// ---- MG-path PCG kernels on quads (level 0, FP32) ------------------------------
// s_new = z + beta s_old; q = A' s_new; alpha = sigma / (s.q)
__global__ void __launch_bounds__(PCG_THREADS) k_spmv_q(const PcgArgs a, Vecs<float> v, MGLev L) {
    __shared__ double scratch[PCG_THREADS];
    pdl_enter();
    if (a.st->done) return;
    const int sc = (a.st->bufsel >> 1) & 1;
    const float beta = (float)a.st->beta;
    const float* so = sc ? v.s[1] : v.s[0];
    float* sn = sc ? v.s[0] : v.s[1];
    Acc<float> sq;
    mg_for_quads<true>(a, L, [&](int x, int y, int z0, long long c0) {
        uint16_t cc[4];
        codes4(a.code, c0, cc);
        if (!any_fluid(cc)) return;
        Q7 zq;
        load_q7(zq, v.z, c0, L, x, y, z0);
        Q7 n = zq;  // s_new around the quad; beta = 0: s = z, s_old is not read
        if (beta != 0.f) {
            Q7 sq7;
            load_q7(sq7, so, c0, L, x, y, z0);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                n.c[i] = zq.c[i] + beta * sq7.c[i];
                n.xp[i] = zq.xp[i] + beta * sq7.xp[i];
                n.xm[i] = zq.xm[i] + beta * sq7.xm[i];
                n.yp[i] = zq.yp[i] + beta * sq7.yp[i];
                n.ym[i] = zq.ym[i] + beta * sq7.ym[i];
            }
            n.zm = zq.zm + beta * sq7.zm;
            n.zp = zq.zp + beta * sq7.zp;
        }
        float qv[4], snc[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (cc[i] & CODE_FLUID) {
                snc[i] = n.c[i];
                qv[i] = (float)code_ns(cc[i]) * n.c[i] - nbsum(n, i, cc[i]);
                sq.add(snc[i] * qv[i]);
            } else {
                snc[i] = 0.f;
                qv[i] = 0.f;
            }
        }
        st4(sn + c0, snc);
        st4(v.q + c0, qv);
    });
    double acc[1] = {sq.value()};
    if (last_block_reduce<1>(acc, 0, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* s = a.st;
            s->alpha = s->sigma / acc[0];
            if (!isfinite(s->alpha)) {
                s->nan = 1;
                s->done = 1;
            }
            s->bufsel ^= 2;
        }
    }
}

// x += alpha s; r_new = r - alpha q; r.r, max|r|; z = r_new / ns, the first red half
// sweep of the V-cycle from zero (the black one follows as a pass of its own: done
// here it needed r_new / ns of every neighbour from r, q and the codes, 90 us at
// 256^3 against 40 + 20)
__global__ void __launch_bounds__(PCG_THREADS) k_update_q(const PcgArgs a, Vecs<float> v, MGLev L) {
    __shared__ double scratch[PCG_THREADS * 2];
    pdl_enter();
    if (a.st->done) return;
    const int rc = a.st->bufsel & 1, sc = (a.st->bufsel >> 1) & 1;
    const float alpha = (float)a.st->alpha;
    const float* ro = rc ? v.r[1] : v.r[0];
    float* rn = rc ? v.r[0] : v.r[1];
    const float* s = sc ? v.s[1] : v.s[0];
    Acc<float> rr;
    float rmax = 0.f;
    mg_for_quads<true>(a, L, [&](int x, int y, int z0, long long c0) {
        uint16_t cc[4];
        codes4(a.code, c0, cc);
        float sv[4], xv[4], rv[4], qv[4], zv[4];
        unpack4(ld4(s + c0), sv);
        unpack4(ld4(v.x + c0), xv);
        unpack4(ld4(ro + c0), rv);
        unpack4(ld4(v.q + c0), qv);
        if (!any_fluid(cc)) return;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            zv[i] = 0.f;
            if (!(cc[i] & CODE_FLUID)) {
                rv[i] = 0.f;
                continue;
            }
            xv[i] += alpha * sv[i];
            rv[i] -= alpha * qv[i];
            rr.add(rv[i] * rv[i]);
            rmax = fmaxf(rmax, fabsf(rv[i]));
            zv[i] = rv[i] * c_rcp[code_ns(cc[i])];
        }
        st4(v.x + c0, xv);
        st4(rn + c0, rv);
        st4(v.z + c0, zv);
    });
    double acc[2] = {rr.value(), (double)rmax};
    if (last_block_reduce<2>(acc, 0x2, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) {
            PcgState* st = a.st;
            st->rr = acc[0];
            st->rmax = acc[1];
            st->it += 1;
            st->bufsel ^= 1;
            const bool conv = (st->tol_mode == FSIM_TOL_ABS_MAX) ? (acc[1] < st->tol_abs) : (acc[0] <= st->tol_rel2);
            st->converged = conv ? 1 : 0;
            if (conv || st->it >= st->max_iters || !isfinite(acc[0])) st->done = 1;
            if (!isfinite(acc[0])) st->nan = 1;
            if (st->fold_enabled && acc[0] < st->fold_drop * st->rr_update) {
                st->need_fold = 1;
                st->done = 1;
            }
        }
    }
}

// dense copies of a coarse level in shared memory: colour test and neighbour sum
// (a closed face is not read: its neighbour may lie outside the array)
__device__ __forceinline__ bool smem_color(uint32_t cc, int color) {
    return (cc & CC_OP) && ((cc & CS_ODD) != 0) == (color != 0);
}
__device__ __forceinline__ float smem_nbsum4(const float* x, int i, uint32_t cc, int sx, int sy) {
    if ((cc & CC_OP) == CC_INTERIOR) return 4.f * (x[i + sx] + x[i - sx] + x[i + sy] + x[i - sy] + x[i + 1] + x[i - 1]);
    float s = 0.f;
    if (cc & 7u) s += coarse_face(cc, 0) * x[i + sx];
    if (cc & (7u << 3)) s += coarse_face(cc, 1) * x[i - sx];
    if (cc & (7u << 6)) s += coarse_face(cc, 2) * x[i + sy];
    if (cc & (7u << 9)) s += coarse_face(cc, 3) * x[i - sy];
    if (cc & (7u << 12)) s += coarse_face(cc, 4) * x[i + 1];
    if (cc & (7u << 15)) s += coarse_face(cc, 5) * x[i - 1];
    return s;
}

// coarsest level: symmetric red-black Gauss-Seidel in shared memory, one CTA
__device__ void mg_bottom_block(const MGLev& L, float* sx, float* sf, uint32_t* sc) {
    const int n = L.nx * L.ny * L.nz;  // dense in shared memory, padded in global
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int z = i % L.nz, t = i / L.nz;
        const long long gi = (long long)t * L.pz + z;
        const int odd = (t / L.ny + t % L.ny + z) & 1;
        sx[i] = 0.f;
        sf[i] = L.f[gi];
        sc[i] = L.ccode[gi] | (odd ? CS_ODD : 0);
    }
    __syncthreads();
    const int sxs = L.ny * L.nz, sys = L.nz;
    for (int pass = 0; pass < 2 * MG_BOTTOM_SWEEPS; pass++) {
        // forward half: red then black; backward half: black then red
        for (int h = 0; h < 2; h++) {
            const int color = (pass < MG_BOTTOM_SWEEPS) ? h : 1 - h;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const uint32_t cc = sc[i];
                if (!smem_color(cc, color)) continue;
                sx[i] = coarse_solve(cc, sf[i], smem_nbsum4(sx, i, cc, sxs, sys));
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) L.x[(long long)(i / L.nz) * L.pz + (i % L.nz)] = sx[i];
}

__global__ void __launch_bounds__(1024) k_mg_bottom(const PcgState* st, MGLev L) {
    pdl_enter();
    if (st->done) return;
    __shared__ float sx[MG_BOTTOM_MAX];
    __shared__ float sf[MG_BOTTOM_MAX];
    __shared__ uint32_t sc[MG_BOTTOM_MAX];
    mg_bottom_block(L, sx, sf, sc);
}

// The coarse part of the V-cycle in one launch: levels lc .. last (lc's rhs was
// restricted by the caller) run by one thread-block cluster, the passes over a
// level separated by cluster barriers (release/acquire at cluster scope, so
// each pass sees the previous pass's global writes).  Replaces ~11 launches per
// level of latency-bound small kernels.
constexpr int MG_MAX_LEVELS = 12;
constexpr int MG_CLUSTER_THREADS = 512;
// Largest level handed to the cluster kernel: 32^3 and its like.  A pass over 32^3
// takes the cluster ~1.3 us and a launch of its own ~3.8; the 64^3 level (262k cells)
// would not fit the cluster's shared memory, and takes 3.9 us a pass in launches.
constexpr long long MG_CLUSTER_CELLS = 60000;
constexpr int MG_CLUSTER_SMEM = 200 * 1024;  // dynamic shared memory limit of the cluster kernel

struct MGChain {
    MGLev lev[MG_MAX_LEVELS];
    int lc, last, nu;
    int ls;  // first level small enough to run in one CTA's shared memory (<= last)
    // levels lc .. ls-1 as x slabs in distributed shared memory (slab != 0):
    // planes per CTA and float offset of each level in the pool, then the offset
    // of rank 0's shared-memory levels
    int slab;
    int P[MG_MAX_LEVELS];
    int off[MG_MAX_LEVELS];
    int soff;
};

// ---- levels in shared memory ----------------------------------------------------
// A level (or a CTA's x slab of one) in shared memory.  Pairs of z-neighbouring
// cells (2j, 2j + 1) hold one cell of either colour, so x, f, the codes and the
// reciprocal diagonals are kept as a red and a black array indexed by pair: a half
// sweep over one colour reads the other colour's array at p, p +- 1, p +- row and
// p +- plane, free of bank conflicts.  x has a guard plane on either side, rows are
// padded to whole pairs, so every neighbour's slot exists and is finite.  A slab's
// guard planes hold its neighbours' boundary planes: whoever writes a boundary
// cell also writes it there (distributed shared memory), and the cluster barrier
// separates the passes.  (The passes copy it: a store to the pool could change the
// shared one.)  The pre-smoothing ends with the black cells and the
// post-smoothing starts with them, so only red cells have a residual and only red
// cells need the coarse correction.
// What bounds it is latency: barriers, shared-memory round trips, and the kernel's own
// instructions.  It runs once per V-cycle between kernels that stream through the
// caches, so its code is fetched anew each time: the passes are small functions shared
// by all levels, not inlined, and only the smoother keeps the operator in registers
// and is unrolled.  From 16^3 down (32^3 grid) / from 32^3 down on a 128^3 and on a
// 256^3 grid: 23, 38 and 51 us; with everything inlined and unrolled 19, 39 and 72;
// with the codes decoded in every pass, both colours in one array and the boundary
// planes read over the cluster, 29, 49 and 68.
constexpr int MG_SMEM_CELLS = 4096;  // padded cells of a level rank 0 runs alone

struct SLev {
    int nx, ny, nz, pr, plane;  // global cells per axis, pairs per row and per plane
    int x0, P, np, n;           // first plane, planes per CTA, planes and pairs held
    int xo, xc;                 // pool offset of red x (black: + xc)
    int fo, fc;                 // red f (black: + fc); then codes, diagonals (red, black) and r
    float *lo, *hi;             // the neighbours' copies of the first / last red plane, or null
};
extern __shared__ float pool[];
__device__ __forceinline__ int slev_co(const SLev& L) { return L.fo + 2 * L.fc; }
__device__ __forceinline__ int slev_do(const SLev& L) { return L.fo + 4 * L.fc; }
__device__ __forceinline__ int slev_ro(const SLev& L) { return L.fo + 6 * L.fc; }

// floats of a level with `planes` planes
__host__ __device__ inline long long slev_floats(int planes, int ny, int nz) {
    const long long plane = (long long)ny * ((nz + 1) / 2);
    return plane * (9ll * planes + 4);
}
__device__ __forceinline__ void slev_make(SLev& L, const MGLev& G, int off, int planes, int x0) {
    L.nx = G.nx; L.ny = G.ny; L.nz = G.nz;
    L.pr = (G.nz + 1) >> 1;
    L.plane = G.ny * L.pr;
    L.x0 = x0;
    L.P = planes;
    L.np = max(0, min(planes, G.nx - x0));
    L.n = L.np * L.plane;
    L.xc = (planes + 2) * L.plane;
    L.fc = planes * L.plane;
    L.xo = off + L.plane;
    L.fo = off + 2 * L.xc;
    L.lo = L.hi = nullptr;
}
// pair p: plane, row, place along z; par: its red cell is at z = 2j + par
__device__ __forceinline__ void slev_pair(const SLev& L, int p, int& xl, int& y, int& j, int& par) {
    const int row = (int)((unsigned)p / (unsigned)L.pr);
    j = p - row * L.pr;
    xl = (int)((unsigned)row / (unsigned)L.ny);
    y = row - xl * L.ny;
    par = (L.x0 + xl + y) & 1;
}

// codes (with the cell's place in its pair) and diagonals from global memory; x, f
// and r to zero (the guard planes too)
__device__ __noinline__ void slev_init(const SLev& SL, const MGLev& G) {
    const SLev L = SL;
    for (int i = threadIdx.x; i < 2 * L.xc; i += blockDim.x) pool[L.xo - L.plane + i] = 0.f;
#pragma unroll 1
    for (int p = threadIdx.x; p < L.n; p += blockDim.x) {
        int xl, y, j, par;
        slev_pair(L, p, xl, y, j, par);
        const uint32_t* row = G.ccode + ((long long)(L.x0 + xl) * G.ny + y) * G.pz + 2 * j;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int e = par ^ c;
            const uint32_t cc = 2 * j + e < L.nz ? row[e] : 0u;
            pool[slev_co(L) + c * L.fc + p] = __uint_as_float(cc | (e ? CS_HIGH : 0u));
            pool[slev_do(L) + c * L.fc + p] =
                is_fluid(cc) ? __fdividef(8.f, small_float((uint32_t)coarse_diag8(cc))) : 0.f;
            pool[L.fo + c * L.fc + p] = 0.f;
        }
        pool[slev_ro(L) + p] = 0.f;
    }
}
__device__ __noinline__ void slev_load_f(const SLev& SL, const MGLev& G) {
    const SLev L = SL;
#pragma unroll 1
    for (int p = threadIdx.x; p < L.n; p += blockDim.x) {
        int xl, y, j, par;
        slev_pair(L, p, xl, y, j, par);
        const float* row = G.f + ((long long)(L.x0 + xl) * G.ny + y) * G.pz + 2 * j;
#pragma unroll
        for (int c = 0; c < 2; c++)
            if (pool[slev_do(L) + c * L.fc + p] != 0.f) pool[L.fo + c * L.fc + p] = row[par ^ c];
    }
}
__device__ __noinline__ void slev_store_x(const SLev& SL, const MGLev& G) {
    const SLev L = SL;
#pragma unroll 1
    for (int p = threadIdx.x; p < L.n; p += blockDim.x) {
        int xl, y, j, par;
        slev_pair(L, p, xl, y, j, par);
        float* row = G.x + ((long long)(L.x0 + xl) * G.ny + y) * G.pz + 2 * j;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int e = par ^ c;
            if (2 * j + e < L.nz) row[e] = pool[L.xo + c * L.xc + p];
        }
    }
}

// sum of (open quarters * neighbour) around the cell of colour c in pair p, from the
// other colour's x (all loads are independent of each other and of the code's)
__device__ __forceinline__ float slev_sum4(const SLev& L, int c, int p, uint32_t cc) {
    const float* o = pool + L.xo + (1 - c) * L.xc + p;
    const float a = o[L.plane], b = o[-L.plane], d = o[L.pr], f = o[-L.pr], m = o[0], lo = o[-1], hi = o[1];
    const float zp = (cc & CS_HIGH) ? hi : m, zm = (cc & CS_HIGH) ? m : lo;
    if ((cc & CC_OP) == CC_INTERIOR) return 4.f * ((a + b) + (d + f) + (zp + zm));
    return (coarse_face(cc, 0) * a + coarse_face(cc, 1) * b) + (coarse_face(cc, 2) * d + coarse_face(cc, 3) * f) +
           (coarse_face(cc, 4) * zp + coarse_face(cc, 5) * zm);
}
__device__ __forceinline__ void slev_put(const SLev& L, int c, int p, float v) {
    pool[L.xo + c * L.xc + p] = v;
    if (L.lo && p < L.plane) L.lo[c * L.xc + p] = v;
    if (L.hi && p >= L.n - L.plane) L.hi[c * L.xc + p - (L.n - L.plane)] = v;
}
// scaled residual of the red cells (the black ones, just updated, have none)
__device__ __noinline__ void slev_resid(const SLev& SL) {
    const SLev L = SL;
#pragma unroll 1
    for (int p = threadIdx.x; p < L.n; p += blockDim.x) {
        const uint32_t cc = __float_as_uint(pool[slev_co(L) + p]);
        if (!is_fluid(cc)) continue;
        pool[slev_ro(L) + p] =
            coarse_resid(cc, pool[L.fo + p], pool[L.xo + p], slev_sum4(L, 0, p, cc)) * coarse_pscale(cc);
    }
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return n;
}
// the same shared-memory location in cluster CTA `rank` (generic address)
template <typename T>
__device__ __forceinline__ T* dsm(T* p, unsigned rank) {
    unsigned long long out;
    asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<unsigned long long>(p)), "r"(rank));
    return reinterpret_cast<T*>(out);
}

// who runs a level: one warp, one CTA or the cluster
enum { SYNC_WARP, SYNC_CTA, SYNC_CLUSTER };
__device__ __forceinline__ void level_sync(int sync) {
    if (sync == SYNC_CLUSTER) cluster_barrier();
    else if (sync == SYNC_CTA) __syncthreads();
    else __syncwarp();
}

// A cell's update in registers.  The six face weights (0, 1/4 .. 1) are three pairs of
// 16-bit floats, which hold them exactly and unpack with one instruction each: an
// update is 7 loads and ~25 instructions, half of what decoding the code takes.
struct SOp {
    uint32_t x, y, z;  // z: the pair's other cell, then the next pair's
    float di, f;       // sign of di: set if the next pair is the one above
};
__device__ __forceinline__ uint32_t face_pair(uint32_t cc, int k) {
    return (__float_as_uint(0.25f * coarse_face(cc, k)) >> 16) | __float_as_uint(0.25f * coarse_face(cc, k + 1));
}
__device__ __forceinline__ SOp slev_op(const SLev& L, int c, int p) {
    const float* fp = pool + L.fo + c * L.fc + p;
    const uint32_t cc = __float_as_uint(fp[2 * L.fc]), z = face_pair(cc, 4);
    const bool high = (cc & CS_HIGH) != 0;
    SOp o;
    o.x = face_pair(cc, 0);
    o.y = face_pair(cc, 2);
    o.z = high ? (z << 16) | (z >> 16) : z;
    o.di = high ? -fp[4 * L.fc] : fp[4 * L.fc];
    o.f = fp[0];
    return o;
}
__device__ __forceinline__ float w_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float w_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ void slev_update(const SLev& L, int c, int p, const SOp& op) {
    const float* o = pool + L.xo + (1 - c) * L.xc + p;
    const float xp = o[L.plane], xm = o[-L.plane], yp = o[L.pr], ym = o[-L.pr], m = o[0];
    const float zn = o[signbit(op.di) ? 1 : -1];
    const float sum = (w_lo(op.x) * xp + w_hi(op.x) * xm) + (w_lo(op.y) * yp + w_hi(op.y) * ym) +
                      (w_lo(op.z) * m + w_hi(op.z) * zn);
    slev_put(L, c, p, fabsf(op.di) * (op.f + sum));
}
// `passes` half sweeps, alternating, colour c first, by nt threads
constexpr int SLEV_PAIRS = 4;  // pairs a thread keeps the operator of
__device__ __noinline__ void level_smooth(const SLev& SL, int passes, int c, int sync, int nt) {
    const SLev L = SL;
    const int t = threadIdx.x;
    if (L.n <= SLEV_PAIRS * nt) {
        SOp op[2][SLEV_PAIRS];
#pragma unroll
        for (int i = 0; i < SLEV_PAIRS; i++) {
            if (t + i * nt >= L.n) break;
            op[0][i] = slev_op(L, c, t + i * nt);
            op[1][i] = slev_op(L, 1 - c, t + i * nt);
        }
#pragma unroll 1
        for (int k = 0; k < passes; k += 2) {
#pragma unroll
            for (int i = 0; i < SLEV_PAIRS; i++) {
                if (t + i * nt >= L.n) break;
                slev_update(L, c, t + i * nt, op[0][i]);
            }
            level_sync(sync);
            if (k + 1 == passes) break;
#pragma unroll
            for (int i = 0; i < SLEV_PAIRS; i++) {
                if (t + i * nt >= L.n) break;
                slev_update(L, 1 - c, t + i * nt, op[1][i]);
            }
            level_sync(sync);
        }
        return;
    }
#pragma unroll 1
    for (int k = 0; k < passes; k++) {
#pragma unroll 1
        for (int p = t; p < L.n; p += nt) slev_update(L, c ^ (k & 1), p, slev_op(L, c ^ (k & 1), p));
        level_sync(sync);
    }
}

__device__ __forceinline__ float fw_weight(int d) { return (d == 0 || d == 1) ? 0.75f : 0.25f; }

// D.f = 0.5 * sum P r over the red fine cells of F.  Fine plane fx lies in cluster CTA
// fx / F.P; D's pairs i0, i0 + step, ... are this thread's, in CTA `drank`.
__device__ __noinline__ void slev_restrict(const SLev& SF, const SLev& SD, int dn, int i0, int step, unsigned drank) {
    const SLev F = SF, D = SD;
    float* f = dsm(pool + D.fo, drank);
    const float* diag = dsm(pool + slev_do(D), drank);
#pragma unroll 1
    for (int i = i0; i < 2 * dn; i += step) {
        const int c = i >= dn, p = i - c * dn;
        if (diag[c * D.fc + p] == 0.f) continue;
        int xl, cy, j, par;
        slev_pair(D, p, xl, cy, j, par);
        const int cx = D.x0 + xl, cz = 2 * j + (par ^ c);
        float sum = 0.f;
#pragma unroll
        for (int dx = -1; dx <= 2; dx++) {
            const int fx = 2 * cx + dx;
            if (fx < 0 || fx >= F.nx) continue;
            const int ro = (int)((unsigned)fx / (unsigned)F.P);
            const float* plane = dsm(pool + slev_ro(F) + (fx - ro * F.P) * F.plane, (unsigned)ro);
#pragma unroll
            for (int dy = -1; dy <= 2; dy++) {
                const int fy = 2 * cy + dy;
                if (fy < 0 || fy >= F.ny) continue;
                // red: dz has the parity of dx + dy; dz = -1, 1 lie in pairs cz - 1 and cz, dz = 0, 2
                // in cz and cz + 1
                const bool odd = ((dx + dy) & 1) != 0;
                const int ja = odd ? cz - 1 : cz;
                const float* r = plane + fy * F.pr + ja;
                const float ra = ja >= 0 ? r[0] : 0.f, rb = ja + 1 < F.pr ? r[1] : 0.f;
                sum += fw_weight(dx) * fw_weight(dy) * (odd ? 0.25f * ra + 0.75f * rb : 0.75f * ra + 0.25f * rb);
            }
        }
        f[c * D.fc + p] = 0.5f * sum;
    }
}

// x += P x_coarse on L's red cells; coarse plane cx lies in cluster CTA cx / D.P
__device__ __noinline__ void slev_prolong(const SLev& SL, const SLev& SD) {
    const SLev L = SL, D = SD;
#pragma unroll 1
    for (int p = threadIdx.x; p < L.n; p += blockDim.x) {
        const uint32_t cc = __float_as_uint(pool[slev_co(L) + p]);
        if (!is_fluid(cc)) continue;
        int xl, y, j, par;
        slev_pair(L, p, xl, y, j, par);
        const int x = L.x0 + xl;
        // z = 2j + par: coarse j with weight 3/4 and j + 1 or j - 1 with 1/4
        const int jn = par ? j + 1 : j - 1;
        float sum = 0.f;
#pragma unroll
        for (int ox = 0; ox < 2; ox++) {
            const int cx = (x >> 1) - 1 + (x & 1) + ox;
            if (cx < 0 || cx >= D.nx) continue;
            const int ro = (int)((unsigned)cx / (unsigned)D.P);
            const float* plane = dsm(pool + D.xo + (cx - ro * D.P) * D.plane, (unsigned)ro);
            const float wx = (x & 1) != ox ? 0.75f : 0.25f;
#pragma unroll
            for (int oy = 0; oy < 2; oy++) {
                const int cy = (y >> 1) - 1 + (y & 1) + oy;
                if (cy < 0 || cy >= D.ny) continue;
                // colour of coarse cell (cx, cy, z): (cx + cy + z) & 1
                const float* row = plane + cy * D.pr;
                const float a = row[((cx + cy + j) & 1) * D.xc + (j >> 1)];
                const float b = jn >= 0 && jn < D.nz ? row[((cx + cy + jn) & 1) * D.xc + (jn >> 1)] : 0.f;
                sum += wx * ((y & 1) != oy ? 0.75f : 0.25f) * (0.75f * a + 0.25f * b);
            }
        }
        slev_put(L, 0, p, pool[L.xo + p] + coarse_pscale(cc) * sum);
    }
}

// levels ls..last in rank 0's shared memory
__device__ __noinline__ void smem_levels_run(const MGChain& C, const SLev* S) {
#pragma unroll 1
    for (int l = C.ls; l < C.last; l++) {
        level_smooth(S[l], 2 * C.nu, 0, SYNC_CTA, blockDim.x);
        slev_resid(S[l]);
        __syncthreads();
        slev_restrict(S[l], S[l + 1], S[l + 1].n, threadIdx.x, blockDim.x, 0);
        __syncthreads();
    }
    // bottom level (at most 64 cells): symmetric Gauss-Seidel in one warp (red, black, ..,
    // black, red; repeating the middle half sweep would change nothing)
    if (threadIdx.x < 32) level_smooth(S[C.last], 4 * MG_BOTTOM_SWEEPS - 1, 0, SYNC_WARP, 32);
    __syncthreads();
#pragma unroll 1
    for (int l = C.last - 1; l >= C.ls; l--) {
        slev_prolong(S[l], S[l + 1]);
        __syncthreads();
        level_smooth(S[l], 2 * C.nu, 1, SYNC_CTA, blockDim.x);
    }
}

__global__ void __launch_bounds__(MG_CLUSTER_THREADS, 1) k_mg_coarse(const PcgArgs A,
                                                                     const __grid_constant__ MGChain C) {
    __shared__ SLev S[MG_MAX_LEVELS];
    const unsigned rank = cluster_rank(), cs = cluster_size();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // this CTA's levels: slabs lc .. ls-1, then (held by rank 0, known to all) ls .. last
    const int first = C.slab ? C.lc : C.ls;
    if (threadIdx.x == 0) {
        int off = C.soff;
        for (int l = first; l <= C.last; l++) {
            if (l >= C.ls) {
                slev_make(S[l], C.lev[l], off, C.lev[l].nx, 0);
                off += (int)slev_floats(C.lev[l].nx, C.lev[l].ny, C.lev[l].nz);
                continue;
            }
            slev_make(S[l], C.lev[l], C.off[l], C.P[l], (int)rank * C.P[l]);
            if (S[l].np > 0) {
                // the previous CTA's slab is full: its upper guard plane follows P planes
                if (rank > 0) S[l].lo = dsm(pool + S[l].xo + C.P[l] * S[l].plane, rank - 1);
                if (rank + 1 < cs && S[l].x0 + S[l].np < S[l].nx) S[l].hi = dsm(pool + S[l].xo - S[l].plane, rank + 1);
            }
        }
    }
    __syncthreads();
    // the codes were written before the solve's first V-cycle: they are loaded while
    // the predecessor drains (the residual in between is an ordinary launch: it starts
    // when they are complete, and nothing after it starts before it is)
    for (int l = first; l <= C.last; l++)
        if (l < C.ls || rank == 0) slev_init(S[l], C.lev[l]);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (A.st->done) return;  // the same value in every CTA of the cluster
    __syncthreads();
    if (C.ls == C.lc) {
        // rank 0 runs every level alone
        if (rank == 0) {
            slev_load_f(S[C.ls], C.lev[C.ls]);
            __syncthreads();
            smem_levels_run(C, S);
            slev_store_x(S[C.ls], C.lev[C.ls]);
        }
        return;
    }
    if (C.slab) {
        slev_load_f(S[C.lc], C.lev[C.lc]);
        cluster_barrier();  // every slab's guard planes are zero before a neighbour writes them
#pragma unroll 1
        for (int l = C.lc; l < C.ls; l++) {
            level_smooth(S[l], 2 * C.nu, 0, SYNC_CLUSTER, blockDim.x);
            slev_resid(S[l]);
            cluster_barrier();
            // into the CTA's own slab, or into rank 0's first level, spread over the cluster
            if (l + 1 < C.ls) slev_restrict(S[l], S[l + 1], S[l + 1].n, threadIdx.x, blockDim.x, rank);
            else slev_restrict(S[l], S[l + 1], S[l + 1].n, rank * blockDim.x + threadIdx.x, cs * blockDim.x, 0);
            cluster_barrier();
        }
        if (rank == 0) smem_levels_run(C, S);
        cluster_barrier();
#pragma unroll 1
        for (int l = C.ls - 1; l >= C.lc; l--) {
            slev_prolong(S[l], S[l + 1]);
            cluster_barrier();
            level_smooth(S[l], 2 * C.nu, 1, SYNC_CLUSTER, blockDim.x);
        }
        // level lc's correction back to global memory (its slab alone: no other
        // CTA reads this CTA's shared memory after the last barrier)
        slev_store_x(S[C.lc], C.lev[C.lc]);
        return;
    }
    // levels lc .. ls-1 in global memory
    const long long i0 = (long long)rank * blockDim.x + threadIdx.x;
    const long long step = (long long)cs * blockDim.x;
    for (int l = C.lc; l < C.ls; l++) {
        const MGLev& L = C.lev[l];
        for (int k = 0; k < C.nu; k++) {
            mg_for_range(L, i0, step, [&](int x, int y, int z0, long long c0) { smooth_quad<false>(L, L.f, 0, k == 0, x, y, z0, c0); });
            cluster_barrier();
            mg_for_range(L, i0, step, [&](int x, int y, int z0, long long c0) { smooth_quad<false>(L, L.f, 1, 0, x, y, z0, c0); });
            cluster_barrier();
        }
        mg_for_range(L, i0, step, [&](int x, int y, int z0, long long c0) { residual_quad<false>(L, L.f, x, y, z0, c0); });
        cluster_barrier();
        const MGLev& Cl = C.lev[l + 1];
        mg_for_range(Cl, i0, step, [&](int x, int y, int z0, long long c0) { restrict_quad(L, Cl, x, y, z0, c0); });
        cluster_barrier();
    }
    if (rank == 0) {
        slev_load_f(S[C.ls], C.lev[C.ls]);
        __syncthreads();
        smem_levels_run(C, S);
        slev_store_x(S[C.ls], C.lev[C.ls]);
    }
    cluster_barrier();
    for (int l = C.ls - 1; l >= C.lc; l--) {
        const MGLev& L = C.lev[l];
        const MGLev& Cl = C.lev[l + 1];
        mg_for_range(L, i0, step, [&](int x, int y, int z0, long long c0) { prolong_quad<false>(L, Cl, x, y, z0, c0); });
        cluster_barrier();
        for (int k = 0; k < C.nu; k++) {
            mg_for_range(L, i0, step, [&](int x, int y, int z0, long long c0) { smooth_quad<false>(L, L.f, 1, 0, x, y, z0, c0); });
            cluster_barrier();
            mg_for_range(L, i0, step, [&](int x, int y, int z0, long long c0) { smooth_quad<false>(L, L.f, 0, 0, x, y, z0, c0); });
            cluster_barrier();
        }
    }
}

// coarse cell kinds: fluid if any child is fluid, else air if any child is air
__global__ void k_mg_coarsen(MGLev F, const uint8_t* fkind, const uint8_t* fflags, MGLev Cl, uint8_t* ckind) {
    pdl_enter();
    const long long n = (long long)Cl.nx * Cl.ny * Cl.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned iu = (unsigned)i, t = iu / (unsigned)Cl.nz, u = t / (unsigned)Cl.ny;
    const int cz = (int)(iu - t * (unsigned)Cl.nz), cy = (int)(t - u * (unsigned)Cl.ny), cx = (int)u;
    const long long ci = ((long long)cx * Cl.ny + cy) * Cl.pz + cz;
    int best = 2;
    for (int o = 0; o < 8; o++) {
        const int fx = 2 * cx + (o >> 2), fy = 2 * cy + ((o >> 1) & 1), fz = 2 * cz + (o & 1);
        if (fx >= F.nx || fy >= F.ny || fz >= F.nz) continue;
        const long long fi = ((long long)fx * F.ny + fy) * F.pz + fz;
        int k;
        if (fkind) k = fkind[fi];
        else k = (F.code[fi] & CODE_FLUID) ? 0 : (fflags[fi] == C_AIR ? 1 : 2);
        best = min(best, k);
    }
    ckind[ci] = (uint8_t)best;
}

// Coarse operator: the Galerkin operator of piecewise-constant interpolation,
// halved (its energy counts a linear profile twice), kept as a 7-point stencil.
// A coarse face carries the mean of its four fine faces, so that faces partly
// closed by solids conduct less; the fine cells' Dirichlet weights (fluid-air
// faces at level 0) add up, halved and bounded, so that a coarse cell that is
// cut by the free surface stays tied to p = 0 as the fine cells are.  Weights
// are rounded to quarters and eighths: both cells of a face round the same
// sum, so the operator stays symmetric.
// FINE: the finer level is level 0 (16-bit codes).
template <bool FINE>
__global__ void k_mg_code(MGLev F, MGLev L, uint32_t* code) {
    pdl_enter();
    const long long n = (long long)L.nx * L.ny * L.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned iu = (unsigned)i, t = iu / (unsigned)L.nz, u = t / (unsigned)L.ny;
    const int z = (int)(iu - t * (unsigned)L.nz), y = (int)(t - u * (unsigned)L.ny), x = (int)u;
    const long long ci = ((long long)x * L.ny + y) * L.pz + z;
    int face[6] = {0, 0, 0, 0, 0, 0}, dir = 0;
#pragma unroll
    for (int o = 0; o < 8; o++) {
        const int ox = o >> 2, oy = (o >> 1) & 1, oz = o & 1;
        const int fx = 2 * x + ox, fy = 2 * y + oy, fz = 2 * z + oz;
        if (fx >= F.nx || fy >= F.ny || fz >= F.nz) continue;
        const long long fi = ((long long)fx * F.ny + fy) * F.pz + fz;
        const int kx = ox ? 0 : 1, ky = oy ? 2 : 3, kz = oz ? 4 : 5;  // the faces this child shares with the coarse cell
        if (FINE) {
            const uint16_t c = F.code[fi];
            if (!(c & CODE_FLUID)) continue;
            face[kx] += 4 * ((c >> kx) & 1);
            face[ky] += 4 * ((c >> ky) & 1);
            face[kz] += 4 * ((c >> kz) & 1);
            dir += 8 * (code_ns(c) - code_nf(c));
        } else {
            const uint32_t c = F.ccode[fi];
            face[kx] += (int)((c >> (3 * kx)) & 7u);
            face[ky] += (int)((c >> (3 * ky)) & 7u);
            face[kz] += (int)((c >> (3 * kz)) & 7u);
            dir += (int)((c >> CC_DIRICHLET) & 31u);
        }
    }
    uint32_t cc = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        int w = (face[k] + 2) >> 2;  // mean of four faces in quarters
        if (face[k] > 0 && w == 0) w = 1;
        cc |= (uint32_t)w << (3 * k);
    }
    cc |= (uint32_t)min((dir + 1) >> 1, DIRICHLET_MAX) << CC_DIRICHLET;
    code[ci] = cc;
    if (!(cc & CC_OP)) L.x[ci] = 0.f;  // no pass writes it; interpolation reads it
}

// interpolation scale of a level's fluid cells from the next level's kinds
// (outside the level = solid).  One thread per coarse cell: its eight children's
// neighbours all lie in the 27 cells around it, mostly none of them solid (one
// thread per fine cell with eight kind reads: 110 us at 256^3).
template <bool FINE>
__global__ void k_mg_pscale(MGLev F, MGLev Cl, const uint8_t* ckind, uint16_t* code, uint32_t* ccode) {
    pdl_enter();
    const long long n = (long long)Cl.nx * Cl.ny * Cl.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned iu = (unsigned)i, t = iu / (unsigned)Cl.nz, u = t / (unsigned)Cl.ny;
    const int cz = (int)(iu - t * (unsigned)Cl.nz), cy = (int)(t - u * (unsigned)Cl.ny), cx = (int)u;
    const long long ci = ((long long)cx * Cl.ny + cy) * Cl.pz + cz;
    if (ckind[ci] != 0) return;  // no fluid child
    unsigned solid = 0;          // bit 9 (dx + 1) + 3 (dy + 1) + dz + 1
#pragma unroll
    for (int k = 0; k < 27; k++) {
        const int x = cx + k / 9 - 1, y = cy + (k / 3) % 3 - 1, z = cz + k % 3 - 1;
        const bool in = x >= 0 && y >= 0 && z >= 0 && x < Cl.nx && y < Cl.ny && z < Cl.nz;
        if (!in || ckind[((long long)x * Cl.ny + y) * Cl.pz + z] == 2) solid |= 1u << k;
    }
    if (!solid) return;
    for (int o = 0; o < 8; o++) {
        const int sx = o >> 2, sy = (o >> 1) & 1, sz = o & 1;
        const int fx = 2 * cx + sx, fy = 2 * cy + sy, fz = 2 * cz + sz;
        if (fx >= F.nx || fy >= F.ny || fz >= F.nz) continue;
        const long long fi = ((long long)fx * F.ny + fy) * F.pz + fz;
        if (FINE ? !is_fluid(code[fi]) : !is_fluid(ccode[fi])) continue;
        // the child's eight coarse neighbours: the parent (weight 3 of 4 per axis) and the
        // cells next to it on the child's side (1 of 4)
        int k = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int ax = q >> 2, ay = (q >> 1) & 1, az = q & 1;
            const int dx = ax ? 2 * sx - 1 : 0, dy = ay ? 2 * sy - 1 : 0, dz = az ? 2 * sz - 1 : 0;
            if (!((solid >> (9 * (dx + 1) + 3 * (dy + 1) + dz + 1)) & 1u)) k += (ax ? 1 : 3) * (ay ? 1 : 3) * (az ? 1 : 3);
        }
        const unsigned s = (unsigned)(64 - k) & 63u;
        if (!s) continue;
        if (FINE) code[fi] = (uint16_t)(code[fi] | ((s & 3u) << 6) | ((s & 0x3Cu) << 9));
        else ccode[fi] |= s << CC_SCALE;
    }
}

// phi += x; x = 0   (fold the FP32 accumulator into the FP64 solution)
__global__ void __launch_bounds__(PCG_THREADS) k_fold(const PcgArgs a, float* x) {
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int xx, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, xx, y, z, c)) continue;
        if (!(a.code[c] & CODE_FLUID)) continue;
        a.phi[c] += (double)x[c];
        x[c] = 0.f;
    }
    // the iteration goes on unless the residual computed next says otherwise
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->done = 0;
        a.st->need_fold = 0;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

int solver_alloc(fsim_ctx* ctx) {
    SolverBufs& S = ctx->sv;
    const GridGeom& g = ctx->g;
    S.nbx = ceil_div(g.nx, BRX);
    S.nby = ceil_div(g.ny, BRY);
    S.nbz = ceil_div(g.nz, BRZ);
    S.nbricks = (long long)S.nbx * S.nby * S.nbz;
    const size_t nc = (size_t)g.ncell;
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.brick_xyz, S.nbricks * sizeof(int4)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.d_nactive, sizeof(int)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.brick_flag, S.nbricks));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.code, nc * sizeof(uint16_t)));
    FSIM_CUDA_TRY(ctx, cudaMemset(S.code, 0, nc * sizeof(uint16_t)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.b, nc * sizeof(double)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.phi, nc * sizeof(double)));
    FSIM_CUDA_TRY(ctx, cudaMemset(S.phi, 0, nc * sizeof(double)));
    // FP32 set: r[2], s[2], z, q, x  (7 arrays, one allocation)
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.r, 7 * nc * sizeof(float)));
    FSIM_CUDA_TRY(ctx, cudaMemset(S.r, 0, 7 * nc * sizeof(float)));
    S.s = S.r + 2 * nc;
    S.z = S.r + 4 * nc;
    S.q = S.r + 5 * nc;
    S.plo = S.r + 6 * nc;
    int bps = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_update<float>, PCG_THREADS, 0);
    if (bps < 1) bps = 1;
    // a pass takes four bricks per block: no more blocks than a grid has bricks for
    S.grid_blocks = (int)std::min<long long>((long long)ctx->num_sms * bps, (S.nbricks + 3) / 4);
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.partials, (size_t)S.grid_blocks * 4 * sizeof(double)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.counter, sizeof(unsigned)));
    FSIM_CUDA_TRY(ctx, cudaMemset(S.counter, 0, sizeof(unsigned)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.st, sizeof(PcgState)));
    FSIM_CUDA_TRY(ctx, cudaMallocHost(&S.st_host, sizeof(PcgState)));
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.guess, nc * sizeof(float)));
    float fill[7][7];
    for (int nf = 0; nf < 7; nf++)
        for (int ns = 0; ns < 7; ns++) fill[nf][ns] = ns > 0 ? (1.f + TAU * (nf - 1)) / ns : 0.f;
    FSIM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_fill, fill, sizeof(fill)));
    float rcp[7];
    for (int ns = 0; ns < 7; ns++) rcp[ns] = ns > 0 ? 1.f / ns : 1.f;
    FSIM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_rcp, rcp, sizeof(rcp)));
    float psc[64];
    for (int i = 0; i < 64; i++) psc[i] = 64.f / (64 - i);
    FSIM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_pscale, psc, sizeof(psc)));
    // multigrid hierarchy: halve (at least once) until every dimension is <= 4
    MGLevelBufs l0;
    l0.nx = g.nx; l0.ny = g.ny; l0.nz = g.nz; l0.pz = g.pz; l0.ncell = g.ncell;
    l0.code = S.code;
    FSIM_CUDA_TRY(ctx, cudaMalloc(&l0.r, nc * sizeof(float)));
    FSIM_CUDA_TRY(ctx, cudaMemset(l0.r, 0, nc * sizeof(float)));
    S.mg.push_back(l0);
    // at least one coarse level, also below a grid of 3 or 4 cells per axis: the bottom
    // kernel reads coarse codes, and the cycle's level 0 computes z.r
    do {
        const MGLevelBufs& f = S.mg.back();
        MGLevelBufs c;
        c.nx = (f.nx + 1) / 2; c.ny = (f.ny + 1) / 2; c.nz = (f.nz + 1) / 2; c.pz = (c.nz + 3) & ~3;
        c.ncell = (long long)c.nx * c.ny * c.pz;
        FSIM_CUDA_TRY(ctx, cudaMalloc(&c.kind, c.ncell));
        FSIM_CUDA_TRY(ctx, cudaMalloc(&c.ccode, c.ncell * sizeof(uint32_t)));
        FSIM_CUDA_TRY(ctx, cudaMalloc(&c.x, c.ncell * sizeof(float)));
        FSIM_CUDA_TRY(ctx, cudaMalloc(&c.f, c.ncell * sizeof(float)));
        FSIM_CUDA_TRY(ctx, cudaMalloc(&c.r, c.ncell * sizeof(float)));
        FSIM_CUDA_TRY(ctx, cudaMemset(c.x, 0, c.ncell * sizeof(float)));
        FSIM_CUDA_TRY(ctx, cudaMemset(c.f, 0, c.ncell * sizeof(float)));
        FSIM_CUDA_TRY(ctx, cudaMemset(c.r, 0, c.ncell * sizeof(float)));
        FSIM_CUDA_TRY(ctx, cudaMemset(c.ccode, 0, c.ncell * sizeof(uint32_t)));
        FSIM_CUDA_TRY(ctx, cudaMemset(c.kind, 2, c.ncell));
        S.mg.push_back(c);
    } while (std::max(S.mg.back().nx, std::max(S.mg.back().ny, S.mg.back().nz)) > 4);
    if ((long long)S.mg.back().nx * S.mg.back().ny * S.mg.back().nz > MG_BOTTOM_MAX) {
        ctx->err = "multigrid coarsest level too large";
        return FSIM_E_INVALID;
    }
    // cluster for the coarse V-cycle: 16 CTAs where the GPU schedules them, else 8
    S.mg_cluster = 0;
    cudaFuncSetAttribute(k_mg_coarse, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_CLUSTER_SMEM);
    for (int cs : {16, 8}) {
        if (cs > 8 && cudaFuncSetAttribute(k_mg_coarse, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                          cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(cs);
        cfg.blockDim = dim3(MG_CLUSTER_THREADS);
        cfg.dynamicSmemBytes = MG_CLUSTER_SMEM;  // the most a launch asks for
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int nclusters = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, k_mg_coarse, &cfg) == cudaSuccess && nclusters > 0) {
            S.mg_cluster = cs;
            break;
        }
        cudaGetLastError();
    }
    return FSIM_OK;
}

static MGLev mg_lev(const SolverBufs& S, int l, const float* f0, const float* f1, float* x0) {
    const MGLevelBufs& b = S.mg[l];
    MGLev L;
    L.nx = b.nx; L.ny = b.ny; L.nz = b.nz; L.pz = b.pz;
    L.code = b.code;
    L.ccode = b.ccode;
    L.r = b.r;
    if (l == 0) {
        L.x = x0; L.f = f0; L.f1 = f1;
    } else {
        L.x = b.x; L.f = b.f; L.f1 = nullptr;
    }
    return L;
}

// per-solve: coarse cell kinds and codes from the fine flags.  Dependent launches, three per
// level: as ordinary ones they were what a solve that is converged from the start paid for
// (64^3: 167 us, now 138; 154 with the earlier two kernels per level).
static void mg_setup(fsim_ctx* ctx) {
    SolverBufs& S = ctx->sv;
    cudaStream_t st = ctx->stream;
    // the residual passes visit only quads with fluid on level 0, the restriction reads all
    cudaMemsetAsync(S.mg[0].r, 0, (size_t)S.mg[0].ncell * sizeof(float), st);
    for (size_t l = 1; l < S.mg.size(); l++) {
        MGLev F = mg_lev(S, (int)l - 1, nullptr, nullptr, nullptr);
        MGLev Cl = mg_lev(S, (int)l, nullptr, nullptr, nullptr);
        const int nb = ceil_div(S.mg[l].ncell, 256);
        launch_pdl(k_mg_coarsen, nb, 256, st, F, l == 1 ? nullptr : S.mg[l - 1].kind, ctx->flags, Cl, S.mg[l].kind);
        if (l == 1) {
            launch_pdl(k_mg_code<true>, nb, 256, st, F, Cl, S.mg[l].ccode);
            launch_pdl(k_mg_pscale<true>, nb, 256, st, F, Cl, S.mg[l].kind, S.code, nullptr);
        } else {
            launch_pdl(k_mg_code<false>, nb, 256, st, F, Cl, S.mg[l].ccode);
            launch_pdl(k_mg_pscale<false>, nb, 256, st, F, Cl, S.mg[l].kind, nullptr, S.mg[l - 1].ccode);
        }
        ctx->launches += 3;
    }
}

// the V-cycle's sweeps: level 0, separately launched coarse levels, cluster levels, and on
// the free-surface band of level 0 (none unless asked for)
struct MGSweeps {
    int fine, coarse, cluster, band;
};
static MGSweeps mg_sweeps(const fsim_params& P) {
    return {P.mg_sweeps > 0 ? P.mg_sweeps : MG_NU_DEFAULT, P.mg_coarse_sweeps > 0 ? P.mg_coarse_sweeps : MG_NU_COARSE_DEFAULT,
            P.mg_cluster_sweeps > 0 ? P.mg_cluster_sweeps : MG_NU_COARSE_DEFAULT,
            P.mg_boundary_sweeps > 0 ? P.mg_boundary_sweeps : 0};
}

// z = V-cycle(r); r is the current PCG residual (r0 or r1 by device state).
// first_fused: the first red half sweep on level 0 was done by k_update_q; dot_mode >= 0: the
// last level-0 sweep also computes z.r and the CG scalars (k_red modes).
static void mg_vcycle(fsim_ctx* ctx, const PcgArgs& A, int l, const float* r0, const float* r1, float* z,
                      bool first_fused, int dot_mode) {
    const MGSweeps sw = mg_sweeps(ctx->prm);
    const int NU = l == 0 ? sw.fine : sw.coarse, NUC = sw.cluster;
    SolverBufs& S = ctx->sv;
    cudaStream_t st = ctx->stream;
    const int G = S.grid_blocks;
    MGLev L = mg_lev(S, l, r0, r1, z);
    const int last = (int)S.mg.size() - 1;
    if (l == last) {
        launch_pdl(k_mg_bottom, 1, 1024, st, A.st, L);
        ctx->launches += 1;
        return;
    }
    if (l > 0 && S.mg_cluster > 0 && (long long)S.mg[l].ncell <= MG_CLUSTER_CELLS && last - l < MG_MAX_LEVELS) {
        MGChain C{};
        for (int k = l; k <= last; k++) C.lev[k - l] = mg_lev(S, k, nullptr, nullptr, nullptr);
        C.lc = 0;
        C.last = last - l;
        C.nu = NUC;
        // the levels from ls on run in shared memory (x, f, r floats + codes per cell)
        // (long thin levels: their guard planes count, and they halve along one axis only)
        C.ls = C.last;
        size_t smem = 0;
        for (int k = C.last; k >= 0; k--) {
            const MGLevelBufs& b = S.mg[l + k];
            const size_t bytes = (size_t)slev_floats(b.nx, b.ny, b.nz) * sizeof(float);
            if ((long long)b.nx * b.ny * ((b.nz + 1) & ~1) > MG_SMEM_CELLS || smem + bytes > (size_t)MG_CLUSTER_SMEM) break;
            smem += bytes;
            C.ls = k;
        }
        // levels lc .. ls-1 as x slabs in the cluster's distributed shared memory
        // when they fit beside rank 0's levels (else they run in global memory)
        size_t slab_floats = 0;
        for (int k = 0; k < C.ls; k++) {
            const MGLevelBufs& b = S.mg[l + k];
            const int P = ceil_div(b.nx, S.mg_cluster);
            C.P[k] = P;
            C.off[k] = (int)slab_floats;
            slab_floats += (size_t)((slev_floats(P, b.ny, b.nz) + 3) & ~3ll);
        }
        const size_t slab_bytes = slab_floats * sizeof(float) + smem;
        C.slab = (C.ls > 0 && slab_bytes <= (size_t)MG_CLUSTER_SMEM) ? 1 : 0;
        C.soff = C.slab ? (int)slab_floats : 0;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(S.mg_cluster);
        cfg.blockDim = dim3(MG_CLUSTER_THREADS);
        cfg.dynamicSmemBytes = C.slab ? slab_bytes : smem;
        cfg.stream = st;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = S.mg_cluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 2;
        cudaLaunchKernelEx(&cfg, k_mg_coarse, A, C);
        ctx->launches += 1;
        return;
    }
    const int nb = l == 0 ? G : std::min(G, ceil_div(S.mg[l].ncell, 256));
    auto smooth = [&](int color, int first) {
        if (l == 0) launch_pdl(k_mg_smooth<true>, nb, PCG_THREADS, st, A, L, color, first);
        else launch_pdl(k_mg_smooth<false>, nb, PCG_THREADS, st, A, L, color, first);
    };
    // the first red half sweep was done by k_update_q (level 0) or the restriction
    for (int k = 0; k < NU; k++) {
        if (k > 0 || !(l > 0 || first_fused)) {
            smooth(0, k == 0);
            ctx->launches += 1;
        }
        smooth(1, 0);
        ctx->launches += 1;
    }
    const int NB = l == 0 ? sw.band : 0;
    auto smooth_band = [&](int color) {
        launch_pdl(k_mg_smooth_bnd, G, PCG_THREADS, st, A, L, (const int4*)S.bnd_quads, (const int*)S.d_nbnd, color);
        ctx->launches += 1;
    };
    for (int k = 0; k < NB; k++) {
        smooth_band(0);
        smooth_band(1);
    }
    if (l == 0) launch_pdl(k_mg_residual<true>, nb, PCG_THREADS, st, A, L);
    else launch_pdl(k_mg_residual<false>, nb, PCG_THREADS, st, A, L);
    MGLev Cl = mg_lev(S, l + 1, nullptr, nullptr, nullptr);
    launch_pdl(k_mg_restrict, std::min(ctx->num_sms * 8, ceil_div(S.mg[l + 1].ncell, 256)), PCG_THREADS, st, A.st, L, Cl,
               S.mg[l + 1].ncell > 32768 ? 1 : 0);
    mg_vcycle(ctx, A, l + 1, nullptr, nullptr, nullptr, false, -1);
    if (l == 0) launch_pdl(k_mg_prolong<true>, nb, PCG_THREADS, st, A, L, Cl);
    else launch_pdl(k_mg_prolong<false>, nb, PCG_THREADS, st, A, L, Cl);
    // the pre-smoothing's band sweeps in reverse order (the V-cycle stays symmetric)
    for (int k = 0; k < NB; k++) {
        smooth_band(1);
        smooth_band(0);
    }
    for (int k = 0; k < NU; k++) {
        smooth(1, 0);
        if (l == 0 && k == NU - 1 && dot_mode >= 0)
            launch_pdl(k_mg_smooth_dot, nb, PCG_THREADS, st, A, L, dot_mode);
        else
            smooth(0, 0);
        ctx->launches += 2;
    }
    ctx->launches += 3;
}

static int alloc_fp64(fsim_ctx* ctx) {
    SolverBufs& S = ctx->sv;
    if (S.r64) return FSIM_OK;
    const size_t nc = (size_t)ctx->g.ncell;
    FSIM_CUDA_TRY(ctx, cudaMalloc(&S.r64, 6 * nc * sizeof(double)));
    FSIM_CUDA_TRY(ctx, cudaMemset(S.r64, 0, 6 * nc * sizeof(double)));
    S.s64 = S.r64 + 2 * nc;
    S.z64 = S.r64 + 4 * nc;
    S.q64 = S.r64 + 5 * nc;
    return FSIM_OK;
}

void solver_free(fsim_ctx* ctx) {
    SolverBufs& S = ctx->sv;
    cudaFree(S.brick_xyz); cudaFree(S.d_nactive); cudaFree(S.brick_flag); cudaFree(S.code);
    cudaFree(S.b); cudaFree(S.phi); cudaFree(S.r); cudaFree(S.r64); cudaFree(S.partials);
    cudaFree(S.counter); cudaFree(S.st); cudaFreeHost(S.st_host); cudaFree(S.guess);
    cudaFree(S.bnd_quads); cudaFree(S.d_nbnd);
    for (int k = 0; k < SolverBufs::kIterGraphs; k++)
        if (S.iter_exec[k]) cudaGraphExecDestroy(S.iter_exec[k]);
    for (size_t l = 0; l < S.mg.size(); l++) {
        cudaFree(S.mg[l].r);
        if (l > 0) {
            cudaFree(S.mg[l].kind); cudaFree(S.mg[l].ccode); cudaFree(S.mg[l].x); cudaFree(S.mg[l].f);
        }
    }
    S = SolverBufs{};
}

// ---- judged initial guess --------------------------------------------------
// ||b - A phi|| (previous pressure) against ||b - A guess||, FP32 per cell and
// FP64 per thread; the last block records which one seeds PCG.
__global__ void __launch_bounds__(PCG_THREADS) k_guess_judge(const PcgArgs a, const float* guess) {
    __shared__ double scratch[PCG_THREADS * 2];
    double acc[2] = {0.0, 0.0};
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        const float ns = (float)code_ns(cc);
        float ap = ns * (float)a.phi[c], ag = ns * guess[c];
#pragma unroll
        for (int k = 0; k < 6; k++)
            if ((cc >> k) & 1) {
                const long long j = c + nb_off(a.B, k);
                ap -= (float)a.phi[j];
                ag -= guess[j];
            }
        const float bc = (float)a.b[c];
        const float rp = bc - ap, rg = bc - ag;
        acc[0] += (double)(rp * rp);
        acc[1] += (double)(rg * rg);
    }
    if (last_block_reduce<2>(acc, 0, a.partials, a.counter, scratch)) {
        if (threadIdx.x == 0) a.st->guess_used = (acc[1] < acc[0]) ? 1 : 0;
    }
}

// r = b - A phi in FP64 on the fluid cells of the active bricks (0 elsewhere):
// the rhs of the correction the previous pressure still needs
__global__ void __launch_bounds__(PCG_THREADS) k_prev_residual(const PcgArgs a, double* r) {
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        const uint16_t cc = a.code[c];
        if (!(cc & CODE_FLUID)) continue;
        double ap = (double)code_ns(cc) * a.phi[c];
#pragma unroll
        for (int k = 0; k < 6; k++)
            if ((cc >> k) & 1) ap -= a.phi[c + nb_off(a.B, k)];
        r[c] = a.b[c] - ap;
    }
}

// guess = phi + correction on the fluid cells of the active bricks
__global__ void __launch_bounds__(PCG_THREADS) k_guess_add_prev(const PcgArgs a, float* guess) {
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        if (a.code[c] & CODE_FLUID) guess[c] = (float)(a.phi[c] + (double)guess[c]);
    }
}

__global__ void __launch_bounds__(PCG_THREADS) k_guess_apply(const PcgArgs a, const float* guess) {
    if (!a.st->guess_used) return;
    const int nact = *a.nactive;
    for (int bk = blockIdx.x; bk < nact; bk += gridDim.x) {
        int x, y, z;
        long long c;
        if (!brick_cell(a.B, a.bxyz[bk], threadIdx.x, x, y, z, c)) continue;
        if (a.code[c] & CODE_FLUID) a.phi[c] = (double)guess[c];
    }
}

template <typename T>
static int run_pcg(fsim_ctx* ctx, PcgArgs& A, Vecs<T> v, int precision, int precond, fsim_step_stats* stats) {
    SolverBufs& S = ctx->sv;
    cudaStream_t st = ctx->stream;
    const int G = S.grid_blocks;
    const bool fold = (precision == FSIM_PREC_MIXED);
    const bool mg = (precond == FSIM_PRECOND_MG) && sizeof(T) == 4;
    int folds = 0;
    auto read_state = [&]() -> int {
        fetch_small(S.st_host, S.st, (int)sizeof(PcgState), st);
        FSIM_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        return FSIM_OK;
    };
    // z = M^-1 r and sigma (mode 0 setup, 1 iteration, 2 after a fold)
    auto precondition = [&](int mode, bool black_done) {
        if (mg) {
            // mode 1: k_update_q already did the first half sweep; the V-cycle ends with z.r
            mg_vcycle(ctx, A, 0, (const float*)(const void*)v.r[0], (const float*)(const void*)v.r[1],
                      (float*)(void*)v.z, mode == 1, mode);
        } else {
            if (!black_done) {
                k_black<T><<<G, PCG_THREADS, 0, st>>>(A, v);
                ctx->launches += 1;
            }
            k_red<T><<<G, PCG_THREADS, 0, st>>>(A, v, mode);
            ctx->launches += 1;
        }
    };
    if (mg) mg_setup(ctx);
    const MGSweeps sw = mg_sweeps(ctx->prm);
    if (mg && sw.band > 0) {
        if (!S.bnd_quads) {
            FSIM_CUDA_TRY(ctx, cudaMalloc(&S.bnd_quads, (size_t)(ctx->g.ncell / 4 + 1) * sizeof(int4)));
            FSIM_CUDA_TRY(ctx, cudaMalloc(&S.d_nbnd, sizeof(int)));
        }
        FSIM_CUDA_TRY(ctx, cudaMemsetAsync(S.d_nbnd, 0, sizeof(int), st));
        k_bnd_list<<<G, PCG_THREADS, 0, st>>>(A, mg_lev(S, 0, nullptr, nullptr, nullptr), S.bnd_quads, S.d_nbnd);
        ctx->launches += 1;
    }
    // initial residual, preconditioned residual, sigma.  k_residual stays an ordinary launch:
    // k_mg_coarse reads the level codes before its dependency wait, which is only safe behind
    // a kernel that starts after the set-up is complete and does not trigger early.
    k_residual<T><<<G, PCG_THREADS, 0, st>>>(A, v, 1, 1);
    ctx->launches += 1;
    precondition(0, false);
    fsim_record(ctx, EV_PCG_SETUP);
    int rc = read_state();
    if (rc) return rc;
    // An iteration is the matrix product and update, and the preconditioner of the next
    // one follows only if there is a next one: [M^-1, A s, update] is a CUDA graph
    // (captured once per context and configuration; every kernel reads its varying
    // scalars from the device state), and the first iteration after the start or a fold,
    // where z is there already, launches its two kernels.  With the preconditioner at
    // the end of each iteration the last one's launches found the solve stopped (about
    // 2 us each), as did those after the last fold: 0.68 -> 0.64 ms at 32^3, 1.43 -> 1.30
    // at 128^3, 3.58 -> 3.38 at 256^3 (dam breaks).
    auto enqueue_product = [&]() {
        if (mg) {
            const MGLev L0 = mg_lev(S, 0, nullptr, nullptr, nullptr);
            Vecs<float> vf = *reinterpret_cast<Vecs<float>*>(&v);
            launch_pdl(k_spmv_q, G, PCG_THREADS, st, A, vf, L0);
            launch_pdl(k_update_q, G, PCG_THREADS, st, A, vf, L0);
        } else {
            k_spmv<T><<<G, PCG_THREADS, 0, st>>>(A, v);
            k_update<T><<<G, PCG_THREADS, 0, st>>>(A, v);
        }
        ctx->launches += 2;
    };
    // (all that the captured launches depend on)
    const std::array<int, 6> key = mg ? std::array<int, 6>{(int)sizeof(T), 1, sw.fine, sw.coarse, sw.cluster, sw.band}
                                      : std::array<int, 6>{(int)sizeof(T), 0, 0, 0, 0, 0};
    int gi = -1;
    for (int k = 0; k < SolverBufs::kIterGraphs; k++)
        if (S.iter_exec[k] && S.iter_key[k] == key) gi = k;
    if (gi < 0) {
        // a free slot, else the least recently used one
        gi = 0;
        for (int k = 0; k < SolverBufs::kIterGraphs; k++) {
            if (!S.iter_exec[k]) { gi = k; break; }
            if (S.iter_used[k] < S.iter_used[gi]) gi = k;
        }
        if (S.iter_exec[gi]) {
            cudaGraphExecDestroy(S.iter_exec[gi]);
            S.iter_exec[gi] = nullptr;
        }
        const long long l0 = ctx->launches;
        cudaGraph_t graph = nullptr;
        FSIM_CUDA_TRY(ctx, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        precondition(1, true);
        enqueue_product();
        FSIM_CUDA_TRY(ctx, cudaStreamEndCapture(st, &graph));
        cudaError_t ie = cudaGraphInstantiate(&S.iter_exec[gi], graph, 0);
        cudaGraphDestroy(graph);
        FSIM_CUDA_TRY(ctx, ie);
        S.iter_key[gi] = key;
        S.iter_kernels[gi] = (int)(ctx->launches - l0);
        ctx->launches = l0;
    }
    S.iter_used[gi] = ++S.iter_clock;
    cudaGraphExec_t iter_exec = S.iter_exec[gi];
    const int iter_kernels = S.iter_kernels[gi];
    double& conv_rate = S.conv_rate[mg ? 1 : 0];
    // Iterations are launched in chunks between host reads of the state.  The
    // chunk is the number of iterations the measured convergence rate (residual
    // norm factor per iteration, carried over from earlier solves) needs to reach
    // the next stop -- the tolerance or the next fold -- so that few iterations
    // are launched past the stop (they exit at once) and few reads are wasted.
    const int chunk_cap = mg ? 16 : 64;
    auto plan = [&]() -> int {
        const PcgState& h = *S.st_host;
        const double rate = conv_rate;
        if (!(rate > 0.0 && rate < 1.0)) return mg ? 2 : 4;
        const double lr = std::log(rate);
        double n = 1e9;
        if (h.tol_mode == FSIM_TOL_ABS_MAX) {
            if (h.rmax > 0.0 && h.tol_abs > 0.0) n = std::log(h.tol_abs / h.rmax) / lr;
        } else if (h.rr > 0.0 && h.tol_rel2 > 0.0) {
            n = 0.5 * std::log(h.tol_rel2 / h.rr) / lr;
        }
        if (fold && h.rr > 0.0 && h.rr_update > 0.0)
            n = std::min(n, 0.5 * std::log(h.fold_drop * h.rr_update / h.rr) / lr);
        return (int)std::min<double>(chunk_cap, std::max(1.0, std::ceil(n)));
    };
    int chunk = plan();
    int it_mark = S.st_host->it;
    double rr_mark = S.st_host->rr;
    bool fresh = true;  // z = M^-1 r is enqueued
    while (!S.st_host->done && !S.st_host->nan) {
        if (fresh) enqueue_product();
        for (int k = fresh ? 1 : 0; k < chunk; k++) {
            FSIM_CUDA_TRY(ctx, cudaGraphLaunch(iter_exec, st));
            ctx->launches += iter_kernels;
        }
        if ((rc = read_state())) return rc;
        fresh = false;
        PcgState& h = *S.st_host;
        if (h.nan) break;
        if (h.done && !h.need_fold && h.it == it_mark) break;  // stopped by the residual after a fold
        if (h.it > it_mark && rr_mark > 0.0 && h.rr > 0.0 && h.rr < rr_mark) {
            const double r = std::pow(h.rr / rr_mark, 0.5 / (h.it - it_mark));
            conv_rate = conv_rate > 0.0 ? 0.5 * (conv_rate + r) : r;
        }
        it_mark = h.it;
        rr_mark = h.rr;
        chunk = plan();
        const bool need_fold = fold && (h.need_fold || h.done);
        if (need_fold && !h.skip) {
            // fold the FP32 correction into the FP64 solution, recompute the true
            // residual in FP64, and restart CG from it (s = M^-1 r, beta = 0)
            k_fold<<<G, PCG_THREADS, 0, st>>>(A, (float*)(void*)v.x);
            k_residual<T><<<G, PCG_THREADS, 0, st>>>(A, v, 0, 0);
            ctx->launches += 2;
            folds++;
            if (h.converged || h.it >= h.max_iters) {
                // expected to be the end: look before launching more
                const int it_before = h.it;
                if ((rc = read_state())) return rc;
                if (!h.done && it_before >= h.max_iters) h.done = 1;
                if (h.done) break;
            } else {
                h.done = 0;
                h.need_fold = 0;
                h.rr_update = h.rr;
            }
            precondition(0, false);
            fresh = true;
            it_mark = h.it;
            rr_mark = h.rr;
            chunk = plan();
        } else if (h.done) {
            break;
        }
    }
    if (precision == FSIM_PREC_FP32) {
        k_fold<<<G, PCG_THREADS, 0, st>>>(A, (float*)(void*)v.x);
        ctx->launches += 2;
        // true residual of the FP32 result (reporting only)
        PcgState& h = *S.st_host;
        const int conv_recursive = h.converged, its = h.it;
        k_residual<T><<<G, PCG_THREADS, 0, st>>>(A, v, 0, 0);
        if ((rc = read_state())) return rc;
        h.it = its;
        h.converged = conv_recursive;
    }
    if (stats) {
        PcgState& h = *S.st_host;
        stats->pcg_iterations = h.it;
        stats->converged = h.converged;
        stats->reliable_updates = folds;
    }
    return FSIM_OK;
}

int solve_pressure(fsim_ctx* ctx, double dt, int precision, int tol_mode, double tol, int max_iters,
                   int warm, fsim_step_stats* stats, const double* rhs_override, int apply) {
    SolverBufs& S = ctx->sv;
    const GridGeom& g = ctx->g;
    cudaStream_t st = ctx->stream;
    const double scale = dt / (ctx->prm.fluid_density * g.hd * g.hd);
    S.last_scale = scale;
    BrickGeo B;
    B.g = g;
    B.nbx = S.nbx; B.nby = S.nby; B.nbz = S.nbz;
    B.sx = (long long)g.pz * g.ny;
    B.sy = g.pz;

    FSIM_CUDA_TRY(ctx, cudaMemsetAsync(S.brick_flag, 0, S.nbricks, st));
    SetupArgs sa;
    sa.B = B;
    sa.flags = ctx->flags;
    for (int a = 0; a < 3; a++) sa.v2[a] = ctx->v2[a];
    sa.avg = ctx->avg;
    const bool learned = warm == FSIM_WARM_LEARNED || warm == FSIM_WARM_LEARNED_RESIDUAL;
    if (learned && !ctx->net) {
        ctx->err = "FSIM_WARM_LEARNED / _LEARNED_RESIDUAL need a network (fsim_set_net)";
        return FSIM_E_STATE;
    }
    // back-off: a network whose guesses keep losing to the previous pressure is
    // skipped (not run) for a growing number of solves
    if (learned && ctx->prm.learned_backoff && ctx->learned_skip > 0) {
        ctx->learned_skip--;
        warm = FSIM_WARM_PREVIOUS;
    }
    // a user or learned guess is judged against the previous pressure after setup
    const bool judged = warm == FSIM_WARM_LEARNED || warm == FSIM_WARM_LEARNED_RESIDUAL ||
                        (warm == FSIM_WARM_GUESS && S.have_guess);
    sa.guess = nullptr;
    sa.rhs_override = rhs_override;
    sa.warm = (warm == FSIM_WARM_ZERO) ? FSIM_WARM_ZERO : FSIM_WARM_PREVIOUS;
    sa.pressure_enabled = ctx->prm.pressure_enabled;
    sa.avg_pressure = ctx->prm.average_pressure;
    sa.pressure_k = ctx->prm.pressure_k;
    sa.inv_h = 1.0 / g.hd;
    sa.inv_scale = 1.0 / scale;
    sa.code = S.code;
    sa.b = S.b;
    sa.phi = S.phi;
    sa.brick_flag = S.brick_flag;
    k_setup<<<ceil_div(g.ncell, 256), 256, 0, st>>>(sa);
    k_compact_bricks<<<1, COMPACT_THREADS, 0, st>>>(S.brick_flag, S.nbricks, S.nby, S.nbz, S.brick_xyz, S.d_nactive);
    ctx->launches += 2;
    fetch_small(&ctx->h_misc[1], S.d_nactive, (int)sizeof(int), st);

    PcgState h{};
    h.tol_mode = tol_mode;
    h.max_iters = max_iters;
    h.tol_abs = tol / scale;
    h.fold_enabled = (precision == FSIM_PREC_MIXED) ? 1 : 0;
    {
        const int d = ctx->prm.refine_digits > 0 ? std::min(ctx->prm.refine_digits, 6) : MIXED_REFINE_DIGITS;
        h.fold_drop = std::pow(10.0, -2.0 * d);  // on r.r
    }
    *S.st_host = h;
    FSIM_CUDA_TRY(ctx, cudaMemcpyAsync(S.st, S.st_host, sizeof(PcgState), cudaMemcpyHostToDevice, st));

    PcgArgs A;
    A.B = B;
    A.bxyz = S.brick_xyz;
    A.nactive = S.d_nactive;
    A.code = S.code;
    A.b = S.b;
    A.phi = S.phi;
    A.st = S.st;
    A.partials = S.partials;
    A.counter = S.counter;
    A.tol_abs = tol / scale;
    A.tol_rel = tol;
    A.skip_bb = rhs_override ? -1.0 : 1e-7 / (scale * scale);
    A.phi_zero = (warm == FSIM_WARM_ZERO && !judged) ? 1 : 0;

    int rc;
    if (judged) {
        fsim_record(ctx, EV_GUESS0);
        if (warm == FSIM_WARM_LEARNED) {
            const long long l0 = ctx->net->launches;
            rc = net_guess(ctx->net, g, S.code, ctx->flags, S.b, S.guess, st);
            ctx->launches += ctx->net->launches - l0;
            if (rc) {
                ctx->err = std::string("warm-start network: ") + fsim_net_last_error(ctx->net);
                return rc;
            }
        } else if (warm == FSIM_WARM_LEARNED_RESIDUAL) {
            // the network answers the residual of the previous pressure; its answer
            // is added to that pressure (FP64 scratch: the FP64 solver's r buffer)
            if ((rc = alloc_fp64(ctx))) return rc;
            FSIM_CUDA_TRY(ctx, cudaMemsetAsync(S.r64, 0, (size_t)g.ncell * sizeof(double), st));
            k_prev_residual<<<S.grid_blocks, PCG_THREADS, 0, st>>>(A, S.r64);
            const long long l0 = ctx->net->launches;
            rc = net_guess(ctx->net, g, S.code, ctx->flags, S.r64, S.guess, st);
            ctx->launches += ctx->net->launches - l0 + 2;
            if (rc) {
                ctx->err = std::string("warm-start network: ") + fsim_net_last_error(ctx->net);
                return rc;
            }
            k_guess_add_prev<<<S.grid_blocks, PCG_THREADS, 0, st>>>(A, S.guess);
        }
        k_guess_judge<<<S.grid_blocks, PCG_THREADS, 0, st>>>(A, S.guess);
        k_guess_apply<<<S.grid_blocks, PCG_THREADS, 0, st>>>(A, S.guess);
        ctx->launches += 2;
        fsim_record(ctx, EV_GUESS1);
    }
    if (precision == FSIM_PREC_FP64) {
        if ((rc = alloc_fp64(ctx))) return rc;
        const size_t nc = (size_t)g.ncell;
        Vecs<double> v;
        v.r[0] = S.r64; v.r[1] = S.r64 + nc;
        v.s[0] = S.s64; v.s[1] = S.s64 + nc;
        v.z = S.z64; v.q = S.q64;
        v.x = S.phi;
        rc = run_pcg<double>(ctx, A, v, precision, FSIM_PRECOND_RBIC, stats);
    } else {
        const size_t nc = (size_t)g.ncell;
        Vecs<float> v;
        v.r[0] = S.r; v.r[1] = S.r + nc;
        v.s[0] = S.s; v.s[1] = S.s + nc;
        v.z = S.z; v.q = S.q;
        v.x = S.plo;
        rc = run_pcg<float>(ctx, A, v, precision, ctx->prm.precond, stats);
    }
    if (rc) return rc;
    PcgState& hs = *S.st_host;
    if (learned && warm != FSIM_WARM_PREVIOUS && ctx->prm.learned_backoff) {
        if (hs.guess_used) {
            ctx->learned_wait = 0;
        } else {
            ctx->learned_wait = ctx->learned_wait ? std::min(2 * ctx->learned_wait, 64) : 1;
            ctx->learned_skip = ctx->learned_wait;
        }
    }
    if (stats) {
        stats->residual_max = hs.rmax * scale;
        stats->residual_rel = hs.bb > 0 ? sqrt(hs.rr / hs.bb) : 0.0;
        stats->rhs_norm = sqrt(hs.bb) * scale;
        stats->num_active_bricks = ctx->h_misc[1];
        stats->guess_used = judged ? (hs.guess_used ? warm : (warm == FSIM_WARM_ZERO ? 0 : FSIM_WARM_PREVIOUS)) : warm;
        stats->ms_guess = 0.f;
        if (judged && ctx->prm.timing) {
            cudaEventSynchronize(ctx->ev[EV_GUESS1]);
            cudaEventElapsedTime(&stats->ms_guess, ctx->ev[EV_GUESS0], ctx->ev[EV_GUESS1]);
        }
    }
    if (hs.nan) {
        ctx->err = "pressure solve produced a non-finite scalar";
        return FSIM_E_NAN;
    }
    if (apply && !hs.skip) launch_apply_pressure(ctx, dt);
    return FSIM_OK;
}

namespace {
__global__ void k_rhs_out(GridGeom g, const double* b, const uint16_t* code, double scale, float* out) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)g.nx * g.ny * g.nz;
    if (j >= n) return;
    const long long c = (j / g.nz) * g.pz + (j % g.nz);
    out[j] = (code[c] & CODE_FLUID) ? (float)(b[c] * scale) : 0.f;
}
}  // namespace

// rhs of the last solve in the reference's units (b = scale * b')
void launch_rhs_out(fsim_ctx* ctx, float* out) {
    const GridGeom& g = ctx->g;
    const long long n = (long long)g.nx * g.ny * g.nz;
    k_rhs_out<<<ceil_div(n, 256), 256, 0, ctx->stream>>>(g, ctx->sv.b, ctx->sv.code, ctx->sv.last_scale, out);
}
