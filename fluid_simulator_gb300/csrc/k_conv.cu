// k_conv.cu -- convolutions of the pressure warm-start network on the
// 5th-generation tensor cores (tcgen05, TMEM accumulators, TMA operands).
//
// Tensors are BF16 in NDHWC order ([n][d][h][w][c], c fastest).  Weights are
// BF16, packed per 8 input channels and N tile (conv_pack_index); accumulation is FP32.
//
// Forward / input-gradient kernels: implicit GEMM
//   D[m, n] = sum_{tap, c} X[voxel(m) + off(tap), c] * W[tap, n, c]
// over output tiles of 8 (w) x 16 (h) x P (d) voxels and NT output channels:
// k_conv_pers (3x3x3 layers) is persistent, one CTA per SM walking the tiles
// with warp-specialized roles (described at the kernel); k_conv_mma (the
// pointwise down-convolutions) gives each CTA one tile.  Per 16-channel chunk
// of the input a CTA loads ONE halo box of the input (10 x 18 x (P + 2) voxels for
// 3x3x3, zero-filled outside the volume, which is the padding) and the chunk's
// weights for all taps (packed in that order, one contiguous copy), in the no-swizzle K-major core-matrix layout (8
// rows x 16 bytes per core matrix, the two 8-channel halves of the chunk in separate
// planes).  A shift by (kh, kw) is a start offset of the A descriptor: row groups of
// 8 voxels are 16-byte rows, ((plane*18 + kh)*10 + kw) * 16 bytes.  One tcgen05.mma
// multiplies the 128 voxels of an input plane by the weights of all three kd side by
// side (M = 128, N = 3 NT, K = 16): its N blocks are the products for the output
// planes pl - 2, pl - 1, pl, whose TMEM column blocks are neighbours.  Input-gradient
// (dgrad) is the same kernel on the output gradient with the per-tap transposed
// weights, (kh, kw) read backwards.  The epilogue reads TMEM with tcgen05.ld, adds the
// bias, applies ReLU or a ReLU-derivative mask, and stores BF16 at a channel
// stride/offset (so encoder outputs land directly in their concatenation slice).
//
// Weight-gradient kernel (k_conv_wgrad): D[(tap, c), n] = sum_v X[v + off(tap), c]
// * G[v, n] with K = voxels, operands in the MN-major layout (described there).
//
// Every wait is bounded; a timeout sets an error bit, waits (bounded) for the
// MMAs already issued, frees TMEM and returns.
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "fsim_ctx.h"
#include "fsim_net.h"

namespace {

constexpr int TW = 8, TH = 16;  // output tile (w, h); M = TW*TH = 128 per plane
constexpr int CONV_THREADS = 128;
constexpr int SMEM_LIMIT = 227 * 1024 - 1024;  // opt-in maximum minus room for static shared memory
constexpr long long SPIN_LIMIT = 1ll << 31;  // clock cycles, about one second

__device__ __forceinline__ unsigned s32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, unsigned phase) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(s32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned phase) {
    const long long t0 = clock64();
    while (!mbar_try(bar, phase))
        if (clock64() - t0 > SPIN_LIMIT) return false;
    return true;
}
__device__ __forceinline__ void tma_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                       uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(s32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(s32(bar))
        : "memory");
}
// contiguous copy; both addresses and the size are multiples of 16 bytes
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s32(dst)),
                 "l"(src), "r"(bytes), "r"(s32(bar))
                 : "memory");
}

// tcgen05 shared-memory matrix descriptor, K-major, no swizzle: core matrices
// of 8 rows x 16 bytes; lbo = byte distance between the two K halves, sbo =
// byte distance between 8-row groups.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version
    return d;                // base offset 0, layout 0 = no swizzle
}
// instruction descriptor: D FP32, A and B BF16, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar))
                 : "memory");
}
// The issuing loops run on the whole warp and let one lane issue (predicated): control
// flow stays uniform, so descriptors live in uniform registers.  With a single thread
// branching off, every MMA first moved its operands there: 48 -> 16 channels at 128^3
// 142 us, now 109; weight gradient of 16 -> 16 at 8 x 64^3 300 us, then 222.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void mma_bf16_one(uint32_t lead, uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void mma_commit_one(uint32_t lead, uint64_t* bar) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(s32(bar)),
        "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, int ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, int ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__host__ __device__ constexpr int tmem_cols(int n) {
    return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512;
}

__device__ __forceinline__ bool bf16_pos(unsigned short bits) { return !(bits & 0x8000u) && bits != 0; }

// ---------------------------------------------------------------------------
// forward / input-gradient
// ---------------------------------------------------------------------------
template <int TAPS, int PLANES>
struct Halo {
    static constexpr int H = TAPS == 27 ? 1 : 0;
    static constexpr int AW = TW + 2 * H, AH = TH + 2 * H, AD = PLANES + 2 * H;
    static constexpr int ROWS = AW * AH * AD;
    static constexpr int KC = ROWS * 16;  // bytes of one 8-channel half
    static constexpr int A_BYTES = 2 * KC;
};

struct MmaArgs {
    int n, d, h, w;      // volume (input and output have the same size)
    int cin, cout, nt;   // nt = output channels per CTA
    int tiles_w, tiles_h, tiles_d, ntiles;
    int stages;
    int flip;            // weights read at tap 26 - t (input gradient)
    const __nv_bfloat16* wgt;   // packed weights (conv_pack_index)
    const float* bias;   // [cout] or null
    int relu;
    const __nv_bfloat16* mask;  // ReLU-derivative mask (out *= mask > 0) or null
    int ms, mo;          // mask channel stride / offset
    __nv_bfloat16* y;
    int ys, yo;          // output channel stride / offset
    unsigned* err;
};

// pointwise (down-)convolutions: one tile of PLANES d-planes per CTA
constexpr int POINT_MAX_STAGES = 8;
template <int PLANES>
__global__ void __launch_bounds__(CONV_THREADS) k_conv_mma(const MmaArgs a, const __grid_constant__ CUtensorMap tx) {
    pdl_enter();
    using G = Halo<1, PLANES>;
    extern __shared__ __align__(128) unsigned char smraw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>(((uintptr_t)smraw + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t full[POINT_MAX_STAGES], empty[POINT_MAX_STAGES], done;
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;

    long long t = blockIdx.x;
    const int nti = (int)(t % a.ntiles);
    t /= a.ntiles;
    const int bw = (int)(t % a.tiles_w);
    t /= a.tiles_w;
    const int bh = (int)(t % a.tiles_h);
    t /= a.tiles_h;
    const int bd = (int)(t % a.tiles_d);
    const int nb = (int)(t / a.tiles_d);
    const int w0 = bw * TW, h0 = bh * TH, d0 = bd * PLANES, n0 = nti * a.nt;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ncols = tmem_cols(PLANES * a.nt);
    const int B_KC = a.nt * 16;
    const int stage_bytes = G::A_BYTES + 2 * B_KC;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_base, ncols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base;

    const int nchunk = a.cin >> 4;
    if (threadIdx.x == 0) {
        const uint32_t idesc = idesc_bf16(a.nt);
        const unsigned tx_bytes = (unsigned)stage_bytes;
        auto issue = [&](int k) {
            const int s = k % a.stages;
            unsigned char* st = sm + s * stage_bytes;
            mbar_expect_tx(&full[s], tx_bytes);
#pragma unroll
            for (int kc = 0; kc < 2; kc++) {
                tma_5d(st + kc * G::KC, &tx, k * 16 + kc * 8, w0 - G::H, h0 - G::H, d0 - G::H, nb, &full[s]);
                bulk_load(st + G::A_BYTES + kc * B_KC, a.wgt + ((long long)(k * 2 + kc) * a.cout + n0) * 8,
                          (unsigned)B_KC, &full[s]);
            }
        };
        bool ok = true;
        const int pre = nchunk < a.stages ? nchunk : a.stages;
        for (int k = 0; k < pre; k++) issue(k);
        int issued = pre, consumed = 0;
        for (int k = 0; k < nchunk; k++) {
            const int s = k % a.stages;
            if (!mbar_wait(&full[s], (unsigned)((k / a.stages) & 1))) { ok = false; break; }
            consumed = k + 1;
            fence_after();
            const uint32_t abase = s32(sm + s * stage_bytes);
            const uint32_t bbase = abase + G::A_BYTES;
            const uint64_t bdesc = sdesc(bbase, (uint32_t)B_KC, 128);
#pragma unroll
            for (int zp = 0; zp < PLANES; zp++) {
                const uint64_t adesc =
                    sdesc(abase + (uint32_t)(zp * G::AH * G::AW * 16), (uint32_t)G::KC, (uint32_t)(G::AW * 16));
                mma_bf16(tmem + (uint32_t)(zp * a.nt), adesc, bdesc, idesc, k > 0 ? 1u : 0u);
            }
            mma_commit(&empty[s]);
            // refill the stage of the chunk before this one: its MMAs have (nearly) finished
            const int b = k - 1;
            if (b >= 0 && b + a.stages < nchunk) {
                if (!mbar_wait(&empty[b % a.stages], (unsigned)((b / a.stages) & 1))) { ok = false; break; }
                issue(b + a.stages);
                issued++;
            }
        }
        mma_commit(&done);
        if (!ok) {
            // let the copies still in flight land before the CTA's shared memory goes away
            for (int k = consumed; k < issued; k++) mbar_wait(&full[k % a.stages], (unsigned)((k / a.stages) & 1));
            s_fail = 1;
            atomicOr(a.err, 1u);
        }
    }
    __syncthreads();
    const bool ok = mbar_wait(&done, 0);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) atomicOr(a.err, 2u);
    } else if (!s_fail) {
        fence_after();
        const int m = warp * 32 + lane;
        const int vw = w0 + (m & 7), vh = h0 + (m >> 3);
#pragma unroll 1
        for (int zp = 0; zp < PLANES; zp++) {
            const int vd = d0 + zp;
            const bool inside = vw < a.w && vh < a.h && vd < a.d;
            const long long vox = (((long long)nb * a.d + vd) * a.h + vh) * a.w + vw;
#pragma unroll 1
            for (int c0 = 0; c0 < a.nt; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(zp * a.nt + c0), r);
                if (!inside) continue;
                const int ch = n0 + c0;
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
                if (a.bias) {
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] += a.bias[ch + j];
                }
                if (a.relu) {
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = fmaxf(v[j], 0.f);
                }
                if (a.mask) {
                    const uint4* mp = reinterpret_cast<const uint4*>(a.mask + vox * a.ms + a.mo + ch);
                    uint4 mv[2] = {mp[0], mp[1]};
                    const unsigned short* mb = reinterpret_cast<const unsigned short*>(mv);
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (!bf16_pos(mb[j])) v[j] = 0.f;
                }
                __align__(16) __nv_bfloat162 o[8];
#pragma unroll
                for (int j = 0; j < 8; j++) o[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                uint4* dst = reinterpret_cast<uint4*>(a.y + vox * a.ys + a.yo + ch);
                dst[0] = reinterpret_cast<const uint4*>(o)[0];
                dst[1] = reinterpret_cast<const uint4*>(o)[1];
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, ncols);
}

// ---------------------------------------------------------------------------
// forward / input-gradient of the 3x3x3 layers: persistent, warp-specialized
// ---------------------------------------------------------------------------
// One CTA per SM walks the output tiles t = blockIdx.x, + gridDim.x, ...  Warp
// 0 (one thread) streams (tile, 16-channel chunk) items into a ring of shared
// memory stages with TMA, warp 1 issues each item's MMAs (nine per input plane) into
// one of two TMEM accumulators, and warps 2-9 drain the other accumulator
// (bias, ReLU or mask, BF16 stores) while the next tile accumulates, so loads,
// MMAs and the epilogue of neighbouring tiles overlap instead of running one
// after the other in every CTA.  When the layer has one N tile and its
// weights fit beside two stages, all chunks' weights are loaded once and stay
// resident; otherwise each stage carries its chunk's weights as above.
// What bounds it: the MMAs' operand reads.  An MMA reads 4 KB of A whatever N is, so
// wide N pays: with one MMA per tap and output plane (N = NT) a 16 -> 16 layer of 128^3
// was 2916 MMAs of 61 cycles per CTA (98 us); with the three kd in one MMA, 1260 of 52
// cycles, and loads (16-byte rows) and stores of the same length beside them: 50 us.
// 48 -> 16: 260 us, now 110, 9% above its MMAs alone.  The sum of an output is taken in
// the same order (chunk, kd, kh, kw).
// Every wait is bounded; a timeout (or a role that gave up) makes all roles
// stop, the copies in flight land, the issued MMAs finish, TMEM is freed.
constexpr int PERS_DRAIN = 8;  // draining warps
constexpr int PERS_THREADS = 64 + 32 * PERS_DRAIN;
constexpr int PERS_MAX_STAGES = 4;

struct PersArgs {
    MmaArgs m;
    int total_tiles;  // tiles_w * tiles_h * tiles_d * n * ntiles
    int wres;         // weights of all chunks resident in shared memory
    int stage_bytes;  // halo box (plus the chunk's weights when not resident)
    int ncols;        // TMEM columns of one accumulator
};

struct TileAt {
    int w0, h0, d0, nb, n0;
};

template <int PLANES>
__device__ __forceinline__ TileAt tile_at(const MmaArgs& a, int t) {
    TileAt c;
    const int nti = t % a.ntiles;
    t /= a.ntiles;
    c.w0 = (t % a.tiles_w) * TW;
    t /= a.tiles_w;
    c.h0 = (t % a.tiles_h) * TH;
    t /= a.tiles_h;
    c.d0 = (t % a.tiles_d) * PLANES;
    c.nb = t / a.tiles_d;
    c.n0 = nti * a.nt;
    return c;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
// bounded wait that also gives up once another role has stopped
__device__ __forceinline__ bool mbar_wait_ab(uint64_t* bar, unsigned phase, volatile int* stop, unsigned* err) {
    const long long t0 = clock64();
    while (!mbar_try(bar, phase)) {
        if (*stop) return false;
        if (clock64() - t0 > SPIN_LIMIT) {
            *stop = 1;
            atomicOr(err, 1u);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

template <int PLANES>
__global__ void __launch_bounds__(PERS_THREADS, 1) k_conv_pers(const PersArgs p,
                                                                const __grid_constant__ CUtensorMap tx) {
    pdl_enter();
    using G = Halo<27, PLANES>;
    const MmaArgs& a = p.m;
    extern __shared__ __align__(128) unsigned char smraw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>(((uintptr_t)smraw + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t full[PERS_MAX_STAGES], empty[PERS_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ __align__(8) uint64_t wfull, done;
    __shared__ uint32_t tmem_base;
    __shared__ int s_stop, s_issued, s_consumed;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int S = a.stages;
    const int nchunk = a.cin >> 4;
    const int B_KC = 27 * a.nt * 16;
    unsigned char* wbase = sm + S * p.stage_bytes;
    const int my_tiles = (int)blockIdx.x < p.total_tiles ? (p.total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int items = my_tiles * nchunk;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], PERS_DRAIN);
        }
        mbar_init(&wfull, 1);
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_stop = 0;
        s_issued = 0;
        s_consumed = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_base, 2 * p.ncols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    volatile int* stop = &s_stop;

    if (warp == 0) {
        if (lane == 0) {
            if (p.wres) {
                mbar_expect_tx(&wfull, (unsigned)(nchunk * 2 * B_KC));
                for (int k = 0; k < 2 * nchunk; k++)
                    bulk_load(wbase + k * B_KC, a.wgt + (long long)k * (B_KC / 2), (unsigned)B_KC, &wfull);
            }
            int issued = 0;
            for (int j = 0; j < items; j++) {
                const int s = j % S;
                if (j >= S && !mbar_wait_ab(&empty[s], (unsigned)(((j / S) - 1) & 1), stop, a.err)) break;
                const TileAt c = tile_at<PLANES>(a, (int)blockIdx.x + (j / nchunk) * (int)gridDim.x);
                const int k = j % nchunk;
                unsigned char* st = sm + s * p.stage_bytes;
                mbar_expect_tx(&full[s], (unsigned)p.stage_bytes);
#pragma unroll
                for (int kc = 0; kc < 2; kc++) {
                    tma_5d(st + kc * G::KC, &tx, k * 16 + kc * 8, c.w0 - 1, c.h0 - 1, c.d0 - 1, c.nb, &full[s]);
                    if (!p.wres)
                        bulk_load(st + G::A_BYTES + kc * B_KC, a.wgt + ((long long)(k * 2 + kc) * a.cout + c.n0) * 27 * 8,
                                  (unsigned)B_KC, &full[s]);
                }
                issued = j + 1;
            }
            s_issued = issued;
        }
    } else if (warp == 1) {
        {
            const uint32_t lead = elect_one() ? 1u : 0u;
            const uint32_t idesc[3] = {idesc_bf16(a.nt), idesc_bf16(2 * a.nt), idesc_bf16(3 * a.nt)};
            const bool ok = !p.wres || __all_sync(0xffffffffu, mbar_wait_ab(&wfull, 0, stop, a.err));
            int consumed = 0;
            for (int j = 0; ok && j < items; j++) {
                const int s = j % S, ti = j / nchunk, k = j % nchunk, buf = ti & 1;
                if (!__all_sync(0xffffffffu, mbar_wait_ab(&full[s], (unsigned)((j / S) & 1), stop, a.err))) break;
                consumed = j + 1;
                if (k == 0 && ti >= 2 &&
                    !__all_sync(0xffffffffu, mbar_wait_ab(&acc_empty[buf], (unsigned)(((ti >> 1) - 1) & 1), stop, a.err)))
                    break;
                fence_after();
                const uint32_t abase = s32(sm + s * p.stage_bytes);
                const uint32_t bbase = p.wres ? s32(wbase + k * 2 * B_KC) : abase + G::A_BYTES;
                // Unrolled, with descriptors formed by adding to two base
                // descriptors (the start-address field is the byte address / 16, so
                // a shift by `row` halo rows adds `row` and a weight row adds 1): one
                // thread issues every MMA of the CTA and must not spend more time
                // per MMA than the tensor core does.
                const uint64_t ad0 = sdesc(abase, (uint32_t)G::KC, (uint32_t)(G::AW * 16));
                const uint64_t bd0 = sdesc(bbase, (uint32_t)B_KC, 128);
                const uint32_t acc0 = tmem + (uint32_t)(buf * p.ncols);
#pragma unroll
                for (int pl = 0; pl < G::AD; pl++) {
                    // input plane pl feeds output planes pl - kd, kd = lo .. hi
                    const int lo = pl >= PLANES ? pl - PLANES + 1 : 0, hi = pl < 2 ? pl : 2;
                    const uint32_t d = acc0 + (uint32_t)((pl - hi) * a.nt);
#pragma unroll
                    for (int g = 0; g < 9; g++) {
                        const uint64_t ad = ad0 + (uint64_t)((pl * G::AH + g / 3) * G::AW + g % 3);
                        const int gw = (a.flip ? 8 - g : g) * 3;
                        const uint64_t bd = bd0 + (uint64_t)((gw + 2 - hi) * a.nt);
                        if (g == 0 && lo == 0 && k == 0) {
                            // output plane pl's first product overwrites, the others add
                            if (hi > 0) mma_bf16_one(lead, d, ad, bd, idesc[hi > 0 ? hi - 1 : 0], 1u);
                            mma_bf16_one(lead, acc0 + (uint32_t)(pl * a.nt), ad, bd0 + (uint64_t)((gw + 2) * a.nt), idesc[0], 0u);
                        } else {
                            mma_bf16_one(lead, d, ad, bd, idesc[hi - lo], 1u);
                        }
                    }
                }
                mma_commit_one(lead, &empty[s]);
                if (k == nchunk - 1) mma_commit_one(lead, &acc_full[buf]);
            }
            if (lane == 0) s_consumed = consumed;
            mma_commit_one(lead, &done);  // arrives once every MMA issued above has completed
        }
    } else {
        const int q = warp & 3;  // the TMEM lane quarter this warp may access
        const int m = q * 32 + lane;
        for (int ti = 0; ti < my_tiles; ti++) {
            const int buf = ti & 1;
            if (!mbar_wait_ab(&acc_full[buf], (unsigned)((ti >> 1) & 1), stop, a.err)) break;
            fence_after();
            const TileAt c = tile_at<PLANES>(a, (int)blockIdx.x + ti * (int)gridDim.x);
            const int vw = c.w0 + (m & 7), vh = c.h0 + (m >> 3);
            const uint32_t lane_addr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * p.ncols);
#pragma unroll 1
            for (int c0 = 0; c0 < a.nt; c0 += 16) {
                const int ch = c.n0 + c0;
                float bias[16];
#pragma unroll
                for (int j = 0; j < 16; j++) bias[j] = a.bias ? a.bias[ch + j] : 0.f;
                // the warps of a lane quarter take every other plane
#pragma unroll 1
                for (int zp = (warp - 2) >> 2; zp < PLANES; zp += PERS_DRAIN / 4) {
                    const int vd = c.d0 + zp;
                    const bool inside = vw < a.w && vh < a.h && vd < a.d;
                    const long long vox = (((long long)c.nb * a.d + vd) * a.h + vh) * a.w + vw;
                    uint4 mv[2] = {};
                    if (a.mask && inside) {
                        const uint4* mp = reinterpret_cast<const uint4*>(a.mask + vox * a.ms + a.mo + ch);
                        mv[0] = mp[0];
                        mv[1] = mp[1];
                    }
                    uint32_t r[16];
                    tmem_ld16(lane_addr + (uint32_t)(zp * a.nt + c0), r);
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
                    if (a.bias) {
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] += bias[j];
                    }
                    if (a.relu) {
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = fmaxf(v[j], 0.f);
                    }
                    if (a.mask) {
                        const unsigned short* mb = reinterpret_cast<const unsigned short*>(mv);
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (!bf16_pos(mb[j])) v[j] = 0.f;
                    }
                    __align__(16) __nv_bfloat162 o[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) o[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                    // lane pairs (neighbours along w) store one voxel's 32 bytes at a time: whole sectors
                    const uint4 lo = reinterpret_cast<const uint4*>(o)[0], hi = reinterpret_cast<const uint4*>(o)[1];
                    const bool odd = (lane & 1) != 0;
                    uint4 x = odd ? lo : hi;
                    x.x = __shfl_xor_sync(0xffffffffu, x.x, 1);
                    x.y = __shfl_xor_sync(0xffffffffu, x.y, 1);
                    x.z = __shfl_xor_sync(0xffffffffu, x.z, 1);
                    x.w = __shfl_xor_sync(0xffffffffu, x.w, 1);
                    const long long v0 = vox - (odd ? 1 : 0);
                    __nv_bfloat16* dst = a.y + v0 * a.ys + a.yo + ch + (odd ? 8 : 0);
                    const bool row = vh < a.h && vd < a.d;
                    if (row && (vw & ~1) < a.w) *reinterpret_cast<uint4*>(dst) = odd ? x : lo;
                    if (row && (vw | 1) < a.w) *reinterpret_cast<uint4*>(dst + a.ys) = odd ? hi : x;
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 32 && !mbar_wait(&done, 0)) atomicOr(a.err, 2u);
    if (threadIdx.x == 0 && s_stop) {
        // let the copies still in flight land before the CTA's shared memory goes away
        for (int j = s_consumed; j < s_issued; j++) mbar_wait(&full[j % S], (unsigned)((j / S) & 1));
        if (p.wres) mbar_wait(&wfull, 0);
    }
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 2 * p.ncols);
}

// ---------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------
// D[(kd, c), n] of tap (kd, kh, kw) = sum over voxels v of X[v + off, c] * G[v, n]:
// K = voxels, and both operands sit in memory with their M / N index (channels)
// contiguous, which is the tensor core's MN-major layout -- TMA boxes are used
// as they land, nothing is transposed.  A tile is 8 (w) x 16 (h) x WG planes of
// voxels; X comes as one box per d-plane, laid out [octet][h][w][8 channels] with
// the halo, so the channel octets of a plane and then of the next planes are
// one equally spaced sequence: with 4 octets (32 input channels) the 16 groups
// of M = 128 are (d-shift kd = 0..2, octet), 12 of them used.  A shift in h or w
// is a start offset, so 9 accumulators (kh, kw) of N columns each cover the 27
// taps.  One MMA takes 16 voxels (two h rows of 8).  Voxels outside the volume are
// zero-filled by TMA (planes outside the sample are fetched at a coordinate
// outside the tensor).  For the pointwise layers the sequence is 16 octets (128
// input channels) of one plane and there is one accumulator.
//
// The tensor core truncates when it adds to its FP32 accumulator, so long chains
// drift: the accumulators are drained into FP32 registers every few planes (864
// MMAs deep, the sums over 2M voxels were 4-6 times less exact than with the
// kernel this one replaced, 215 deep; at 64 they are more exact).  They come in
// parts (the three kh; pointwise: even and odd planes), each drained by its
// own four warps while the other parts' MMAs run.  One CTA per SM: warps 0-11 drain
// and finally add to the gradient, warp 12 streams tiles through two stages, warp
// 13 issues the MMAs.  Every wait is bounded, as in k_conv_pers.
// What bounds it: the MMAs' operand reads, 4 KB of A per MMA whatever N is (~50 cycles).
// With 16 output channels N is two neighbouring planes of G: X planes z .. z + 3 fill
// M = 128, and the block of X plane p and G plane z belongs to kd = p - z (16 -> 16 at
// 8 x 64^3: 222 us with one plane, 112 with two).  Training pass of 8 x 64^3:
// 15.8 ms of weight gradients with the kernel this one replaced (threads
// transposing 27 shifted copies of X into shared memory, two bytes at a time).
constexpr int WG_THREADS = 448;  // 12 draining warps, TMA, MMA
template <int TAPS>
struct Wg {
    static constexpr int H = TAPS == 27 ? 1 : 0;
    static constexpr int OCT = TAPS == 27 ? 4 : 16;     // octets of one X chunk
    static constexpr int PD = TAPS == 27 ? 4 : 2;       // planes of a tile
    static constexpr int XW = TW + 2 * H, XH = TH + 2 * H, XD = PD + 2 * H;
    static constexpr int X_OCT = XW * XH * 16;          // bytes of one octet of a plane
    static constexpr int X_PLANE = OCT * X_OCT;
    static constexpr int X_BYTES = XD * X_PLANE;
    static constexpr int G_OCT = TW * TH * 16;
    static constexpr int ACC = TAPS == 27 ? 9 : 1;      // accumulators (kh, kw)
    static constexpr int PARTS = TAPS == 27 ? 3 : 2;    // groups of accumulators drained apart: kh; even / odd planes
    static constexpr int PACC = TAPS == 27 ? 3 : 1;     // accumulators of a part
};

// planes of G side by side in an MMA's N (see below)
template <int TAPS, int NT>
constexpr int wgrad_zp = TAPS == 27 && NT == 16 ? 2 : 1;

struct WgArgs {
    int cin, cout;
    int n, d, h, w;
    int tiles_w, tiles_h, tiles_d, tiles;
    int nchunk, nparts, ksplit;
    int interval;            // steps (planes or pairs of planes) per drain of an accumulator
    int stage_bytes, ncols;
    float* dw;               // [taps][cout][cin], accumulated
    unsigned* err;
};

// both operands MN-major (bits 15, 16)
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int n) { return idesc_bf16(n) | (1u << 15) | (1u << 16); }
// MN-major, no swizzle: lbo = bytes between 8-voxel groups (K), sbo = between
// 8-channel groups (M / N); inside a group a voxel's 8 channels are 16 bytes
__device__ __forceinline__ uint64_t sdesc_mn(uint32_t saddr, uint32_t lbo, uint32_t sbo) { return sdesc(saddr, lbo, sbo); }

// drains part `pt` of the accumulators `uses` times into registers, then adds them to the gradient
template <int TAPS, int NT>
__device__ __forceinline__ void wgrad_drain(const WgArgs& a, uint32_t tmem, int pt, int uses, int chunk, int cpart,
                                            uint64_t* acc_full, uint64_t* acc_empty, volatile int* stop) {
    using W = Wg<TAPS>;
    constexpr int ZP = wgrad_zp<TAPS, NT>, NC = ZP * NT, COLS = W::PACC * NC;
    const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3;
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(pt * COLS);
    float r[COLS];
#pragma unroll
    for (int k = 0; k < COLS; k++) r[k] = 0.f;
    for (int u = 0; u < uses; u++) {
        if (!mbar_wait_ab(acc_full, (unsigned)(u & 1), stop, a.err)) return;
        fence_after();
#pragma unroll
        for (int c0 = 0; c0 < COLS; c0 += 32) {
            uint32_t v0[16], v1[16];
            tmem_ld16_async(taddr + (uint32_t)c0, v0);
            if (c0 + 16 < COLS) tmem_ld16_async(taddr + (uint32_t)(c0 + 16), v1);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; j++) {
                r[c0 + j] += __uint_as_float(v0[j]);
                if (c0 + 16 < COLS) r[c0 + 16 + j] += __uint_as_float(v1[j]);
            }
        }
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
    }
    // row m = (X plane, octet, channel), column block z = G plane: kd = X plane - z; blocks with
    // another kd hold sums nobody needs
    const int m = q * 32 + lane;
    const int xp = (m >> 3) / W::OCT, c = chunk * W::OCT * 8 + ((m >> 3) % W::OCT) * 8 + (m & 7);
    if (c >= a.cin) return;
#pragma unroll
    for (int z = 0; z < ZP; z++) {
        const int kd = xp - z;
        if (kd < 0 || kd >= (TAPS == 27 ? 3 : 1)) continue;
#pragma unroll
        for (int k = 0; k < W::PACC; k++) {
            const int tap = TAPS == 27 ? kd * 9 + pt * 3 + k : 0;
            float* o = a.dw + ((long long)tap * a.cout + cpart * NT) * a.cin + c;
#pragma unroll
            for (int j = 0; j < NT; j++) atomicAdd(o + (long long)j * a.cin, r[k * NC + z * NT + j]);
        }
    }
}

template <int TAPS, int NT>
__global__ void __launch_bounds__(WG_THREADS, 1) k_conv_wgrad(const WgArgs a, const __grid_constant__ CUtensorMap tx,
                                                              const __grid_constant__ CUtensorMap tg) {
    pdl_enter();
    using W = Wg<TAPS>;
    constexpr int G_PLANE = (NT >> 3) * W::G_OCT;
    constexpr int ZP = wgrad_zp<TAPS, NT>, NC = ZP * NT;
    extern __shared__ __align__(128) unsigned char smraw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>(((uintptr_t)smraw + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t full[2], empty[2], acc_full[3], acc_empty[3], done;
    __shared__ uint32_t tmem_base;
    __shared__ int s_stop, s_issued, s_consumed;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int chunk = (int)blockIdx.x % a.nchunk;
    const int part = ((int)blockIdx.x / a.nchunk) % a.nparts;
    const int ks = (int)blockIdx.x / (a.nchunk * a.nparts);
    const int my_tiles = (a.tiles - 1 - ks) / a.ksplit + 1;  // ks < ksplit <= tiles
    const int steps = my_tiles * (W::PD / ZP);

    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; q++) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < W::PARTS; q++) {
            mbar_init(&acc_full[q], 1);
            mbar_init(&acc_empty[q], 4);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_stop = 0;
        s_issued = 0;
        s_consumed = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_base, a.ncols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    volatile int* stop = &s_stop;

    if (warp == 12) {
        if (lane == 0) {
            int issued = 0;
            for (int j = 0; j < my_tiles; j++) {
                const int q = j & 1;
                if (j >= 2 && !mbar_wait_ab(&empty[q], (unsigned)(((j >> 1) - 1) & 1), stop, a.err)) break;
                int t = ks + j * a.ksplit;
                const int w0 = (t % a.tiles_w) * TW;
                t /= a.tiles_w;
                const int h0 = (t % a.tiles_h) * TH;
                t /= a.tiles_h;
                const int d0 = (t % a.tiles_d) * W::PD, nb = t / a.tiles_d;
                unsigned char* st = sm + q * a.stage_bytes;
                mbar_expect_tx(&full[q], (unsigned)(W::X_BYTES + W::PD * G_PLANE));
                for (int z = 0; z < W::XD; z++) {
                    const int dd = d0 + z - W::H;
                    const bool in = dd >= 0 && dd < a.d;
                    tma_5d(st + z * W::X_PLANE, &tx, 0, w0 - W::H, h0 - W::H, chunk * W::OCT,
                           in ? nb * a.d + dd : a.n * a.d, &full[q]);
                }
                for (int z = 0; z < W::PD; z++) {
                    const int dd = d0 + z;
                    tma_5d(st + W::X_BYTES + z * G_PLANE, &tg, 0, w0, h0, part * (NT >> 3),
                           dd < a.d ? nb * a.d + dd : a.n * a.d, &full[q]);
                }
                issued = j + 1;
            }
            s_issued = issued;
        }
    } else if (warp == 13) {
        {
            const uint32_t lead = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc = idesc_bf16_mn(NC);
            int consumed = 0;
            bool ok = true;
            for (int j = 0; ok && j < my_tiles; j++) {
                const int q = j & 1;
                if (!__all_sync(0xffffffffu, mbar_wait_ab(&full[q], (unsigned)((j >> 1) & 1), stop, a.err))) break;
                consumed = j + 1;
                fence_after();
                const uint32_t xb = s32(sm + q * a.stage_bytes), gb = xb + W::X_BYTES;
                const uint64_t ad0 = sdesc_mn(xb, W::XW * 16, W::X_OCT);
                const uint64_t bd0 = sdesc_mn(gb, TW * 16, W::G_OCT);
#pragma unroll 1
                for (int z = 0; ok && z < W::PD; z += ZP) {
                    const int p = (j * W::PD + z) / ZP;  // pointwise: plane p >> 1 of part p & 1
                    // start-address fields are in 16-byte units
                    const uint64_t adz = ad0 + (uint64_t)(z * W::X_PLANE / 16);
                    const uint64_t bdz = bd0 + (uint64_t)(z * G_PLANE / 16);
#pragma unroll 1
                    for (int pt = 0; pt < W::PARTS; pt++) {
                        if (TAPS == 1 && (p & 1) != pt) continue;
                        const int pp = TAPS == 1 ? p >> 1 : p, np = TAPS == 1 ? (steps + 1 - pt) / 2 : steps;
                        const int use = pp / a.interval, at = pp - use * a.interval;
                        if (at == 0 && use > 0 &&
                            !__all_sync(0xffffffffu,
                                        mbar_wait_ab(&acc_empty[pt], (unsigned)((use - 1) & 1), stop, a.err))) {
                            ok = false;
                            break;
                        }
                        fence_after();
                        const uint64_t adp = adz + (uint64_t)(TAPS == 27 ? pt * W::XW : 0);  // kh = pt
                        const uint32_t acc0 = tmem + (uint32_t)(pt * W::PACC * NC);
#pragma unroll
                        for (int hp = 0; hp < TH / 2; hp++)
#pragma unroll
                            for (int k = 0; k < W::PACC; k++)  // kw = k
                                mma_bf16_one(lead, acc0 + (uint32_t)(k * NC), adp + (uint64_t)(2 * hp * W::XW + k),
                                         bdz + (uint64_t)(2 * hp * TW), idesc, (hp > 0 || at > 0) ? 1u : 0u);
                        if (at == a.interval - 1 || pp == np - 1) mma_commit_one(lead, &acc_full[pt]);
                    }
                }
                mma_commit_one(lead, &empty[q]);
            }
            if (lane == 0) s_consumed = ok ? consumed : -1;
            mma_commit_one(lead, &done);  // arrives once every MMA issued above has completed
        }
    } else if (warp < 4 * W::PARTS) {
        const int pt = warp >> 2;
        const int np = TAPS == 27 ? steps : (steps + 1 - pt) / 2;
        wgrad_drain<TAPS, NT>(a, tmem, pt, (np + a.interval - 1) / a.interval, chunk, part, &acc_full[pt],
                              &acc_empty[pt], stop);
    }
    __syncthreads();
    const bool fin = mbar_wait(&done, 0);
    if (__syncthreads_or(!fin || s_stop || s_consumed != my_tiles) && threadIdx.x == 0) {
        atomicOr(a.err, 4u);
        // let the copies still in flight land before the CTA's shared memory goes away
        for (int j = s_issued > 2 ? s_issued - 2 : 0; j < s_issued; j++)
            mbar_wait(&full[j & 1], (unsigned)((j >> 1) & 1));
    }
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, a.ncols);
}

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

int pick_nt(int cout, int ntmax) {
    if (cout <= ntmax) return cout;
    for (int nt = ntmax; nt >= 16; nt -= 16)
        if (cout % nt == 0) return nt;
    return 16;
}

}  // namespace

static int sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!sms[dev] && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms[dev];
}

// stages of a 3x3x3 tile of `planes` planes and nt output channels that fit in
// shared memory; wres: the weights of all chunks stay resident
static int pers_stages(int planes, int nt, int cin, int cout, bool& wres, int& stage_bytes) {
    const int A = 2 * (TW + 2) * (TH + 2) * (planes + 2) * 16, B = 2 * 27 * nt * 16, room = SMEM_LIMIT - 128;
    const long long w_all = (long long)(cin / 16) * B;
    wres = nt == cout && w_all + 2 * A <= room;
    stage_bytes = wres ? A : A + B;
    const int n = wres ? (int)((room - w_all) / A) : room / stage_bytes;
    return n < PERS_MAX_STAGES ? n : PERS_MAX_STAGES;
}

// The tile with the least estimated time: waves of tiles over the SMs times the MMAs of
// one.  Deep tiles read fewer input planes per output plane (8: 10, 2: 4), so they win
// wherever they fill the chip; on the small coarse layers shallow tiles and fewer
// channels per CTA give it more CTAs (64 -> 64 channels at 16^3: 8 CTAs of 4 planes x 64
// channels 24 us, 64 of 2 x 16 10 us; at 32^3: 64 CTAs of 4 planes 24, 128 of 2 14).
ConvTile conv_tile(int taps, int n, int d, int h, int w, int cin, int cout) {
    const int sms = sm_count() > 0 ? sm_count() : 1;
    if (taps != 27) {
        // pointwise: a plane at a time and fewer channels per CTA until every SM has two
        // tiles (512 -> 64 channels at 16^3: 8 CTAs 28 us, 128 22)
        ConvTile t{4, pick_nt(cout, 128)};
        auto ctas = [&] {
            return (long long)ceil_div(w, TW) * ceil_div(h, TH) * ceil_div(d, t.planes) * n * (cout / t.nt);
        };
        if (ctas() < 2 * sms) t.planes = 1;
        while (ctas() < sms && t.nt % 32 == 0) t.nt /= 2;
        return t;
    }
    ConvTile best{0, 0};
    double least = 0.0;
    for (int planes : {8, 4, 2}) {
        for (int nt = pick_nt(cout, 64); nt >= 16; nt -= 16) {
            bool wres;
            int bytes;
            if (cout % nt || 2 * tmem_cols(planes * nt) > 512 || pers_stages(planes, nt, cin, cout, wres, bytes) < 2)
                continue;
            // cycles of an MMA of N columns (its operands at ~100 bytes a cycle), of the box's
            // 16-byte rows
            auto mma = [](int N) { return 39.0 + 0.31 * N; };
            const double mmas = 9.0 * (2 * mma(nt) + 2 * mma(2 * nt) + (planes - 2) * mma(3 * nt));
            const double rows = 1.2 * 2 * (TW + 2) * (TH + 2) * (planes + 2), item = mmas > rows ? mmas : rows;
            const long long tiles =
                (long long)ceil_div(w, TW) * ceil_div(h, TH) * ceil_div(d, planes) * n * (cout / nt);
            const double cost = (double)((tiles + sms - 1) / sms) * (item * (cin / 16)) + 400.0 * planes;
            if (!best.planes || cost < least) {
                best = ConvTile{planes, nt};
                least = cost;
            }
        }
    }
    return best;
}

// activations [n][d][h][w][c] bf16 read in halo boxes of 8 channels and `planes` output planes
bool conv_act_map(CUtensorMap* m, const void* base, int n, int d, int h, int w, int c, int taps, int planes) {
    auto enc = encoder();
    if (!enc || (reinterpret_cast<uintptr_t>(base) & 15) || c % 16) return false;
    const int H = taps == 27 ? 1 : 0;
    cuuint64_t dims[5] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)d, (cuuint64_t)n};
    cuuint64_t str[4] = {(cuuint64_t)c * 2, (cuuint64_t)c * 2 * w, (cuuint64_t)c * 2 * w * h,
                         (cuuint64_t)c * 2 * w * h * d};
    cuuint32_t box[5] = {8, (cuuint32_t)(TW + 2 * H), (cuuint32_t)(TH + 2 * H), (cuuint32_t)(planes + 2 * H), 1};
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, str, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// weight-gradient operands: [n*d][h][w][c] bf16 with the channel octets as a
// dimension of their own, so that a box holds [octet][h][w][8 channels] of a plane
static bool wgrad_map(CUtensorMap* m, const void* base, long long planes, int h, int w, int c, int oct, int bw, int bh) {
    auto enc = encoder();
    if (!enc || (reinterpret_cast<uintptr_t>(base) & 15) || c % 16) return false;
    cuuint64_t dims[5] = {8, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)(c / 8), (cuuint64_t)planes};
    cuuint64_t str[4] = {(cuuint64_t)c * 2, (cuuint64_t)c * 2 * w, 16, (cuuint64_t)c * 2 * w * h};
    cuuint32_t box[5] = {8, (cuuint32_t)bw, (cuuint32_t)bh, (cuuint32_t)oct, 1};
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, str, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool wgrad_x_map(CUtensorMap* m, const void* base, int n, int d, int h, int w, int c, int taps) {
    return taps == 27 ? wgrad_map(m, base, (long long)n * d, h, w, c, Wg<27>::OCT, Wg<27>::XW, Wg<27>::XH)
                      : wgrad_map(m, base, (long long)n * d, h, w, c, Wg<1>::OCT, Wg<1>::XW, Wg<1>::XH);
}
// output channels per CTA: nine accumulators of nt columns share TMEM with 3x3x3 taps
static int wgrad_nt(int taps, int cout) {
    if (taps == 1 || cout <= 32) return cout;
    return cout % 32 == 0 ? 32 : 16;
}
bool wgrad_g_map(CUtensorMap* m, const void* base, int n, int d, int h, int w, int c, int taps) {
    return wgrad_map(m, base, (long long)n * d, h, w, c, wgrad_nt(taps, c) / 8, TW, TH);
}

template <int PLANES>
static int launch_pointwise(MmaArgs& a, unsigned grid, const ConvLaunch& L, cudaStream_t s) {
    const int nchunk = a.cin / 16, stage = Halo<1, PLANES>::A_BYTES + 2 * a.nt * 16;
    if (stage + 128 > SMEM_LIMIT) return FSIM_E_INVALID;
    // as many CTAs per SM as TMEM holds accumulators of, at most four, with two to eight
    // pipeline stages each (the issuing loop refills a stage one chunk late): their loads, MMAs and epilogues overlap (one CTA per SM took 41 us
    // for 128 -> 32 channels at 64^3, now 27)
    const int fit = 512 / tmem_cols(PLANES * a.nt), ctas = fit < 4 ? fit : 4, room = SMEM_LIMIT / ctas - 1024;
    a.stages = 1;
    while (a.stages < POINT_MAX_STAGES && a.stages < nchunk && (a.stages + 1) * stage + 128 <= room) a.stages++;
    if (a.stages < 2 && nchunk > 1) return FSIM_E_INVALID;
    int smem = a.stages * stage + 128;
    const int least = SMEM_LIMIT / (ctas + 1) + 1024;  // no more CTAs than that
    if (smem < least) smem = least;
    if (set_smem_limit((const void*)k_conv_mma<PLANES>, SMEM_LIMIT) != cudaSuccess) return FSIM_E_CUDA;
    launch_dep(k_conv_mma<PLANES>, grid, CONV_THREADS, smem, s, a, *L.mx);
    return cudaGetLastError() == cudaSuccess ? FSIM_OK : FSIM_E_CUDA;
}

template <int PLANES>
static int launch_pers(const PersArgs& p, int ctas, int smem, const ConvLaunch& L, cudaStream_t s) {
    if (set_smem_limit((const void*)k_conv_pers<PLANES>, SMEM_LIMIT) != cudaSuccess) return FSIM_E_CUDA;
    launch_dep(k_conv_pers<PLANES>, ctas, PERS_THREADS, smem, s, p, *L.mx);
    return cudaGetLastError() == cudaSuccess ? FSIM_OK : FSIM_E_CUDA;
}

int launch_conv_mma(const ConvLaunch& L, cudaStream_t s) {
    const int taps = L.taps;
    if ((taps != 27 && taps != 1) || L.cin % 16 || L.cout % 16 || L.cin <= 0 || L.cout <= 0) return FSIM_E_INVALID;
    if (reinterpret_cast<uintptr_t>(L.wgt) & 15) return FSIM_E_INVALID;  // (bulk copies)
    if (L.ys % 8 || L.yo % 8 || (L.mask && (L.ms % 8 || L.mo % 8))) return FSIM_E_INVALID;
    MmaArgs a{};
    a.n = L.n; a.d = L.d; a.h = L.h; a.w = L.w;
    a.cin = L.cin; a.cout = L.cout;
    const ConvTile tile = conv_tile(taps, L.n, L.d, L.h, L.w, L.cin, L.cout);
    a.nt = tile.nt;
    a.tiles_w = ceil_div(L.w, TW);
    a.tiles_h = ceil_div(L.h, TH);
    a.tiles_d = ceil_div(L.d, tile.planes);
    a.ntiles = L.cout / a.nt;
    a.flip = L.flip;
    a.wgt = L.wgt;
    a.bias = L.bias;
    a.relu = L.relu;
    a.mask = L.mask; a.ms = L.ms; a.mo = L.mo;
    a.y = L.y; a.ys = L.ys; a.yo = L.yo;
    a.err = L.err;
    const long long grid = (long long)a.tiles_w * a.tiles_h * a.tiles_d * L.n * a.ntiles;
    if (grid <= 0) return FSIM_OK;
    const int nchunk = L.cin / 16;
    if (taps == 27) {
        if (grid >= (1ll << 31)) return FSIM_E_INVALID;
        PersArgs p{};
        bool wres;
        p.total_tiles = (int)grid;
        p.ncols = tmem_cols(tile.planes * a.nt);
        a.stages = pers_stages(tile.planes, a.nt, L.cin, L.cout, wres, p.stage_bytes);
        p.wres = wres ? 1 : 0;
        p.m = a;
        int smem = a.stages * p.stage_bytes + (wres ? nchunk * 2 * 27 * a.nt * 16 : 0) + 128;
        if (smem < SMEM_LIMIT / 2 + 1024) smem = SMEM_LIMIT / 2 + 1024;  // one CTA per SM
        const int sms = sm_count();
        if (!sms) return FSIM_E_CUDA;
        const int ctas = grid < sms ? (int)grid : sms;
        return tile.planes == 8   ? launch_pers<8>(p, ctas, smem, L, s)
               : tile.planes == 4 ? launch_pers<4>(p, ctas, smem, L, s)
                                  : launch_pers<2>(p, ctas, smem, L, s);
    }
    return tile.planes == 4 ? launch_pointwise<4>(a, (unsigned)grid, L, s) : launch_pointwise<1>(a, (unsigned)grid, L, s);
}

template <int TAPS, int NT>
static int launch_wgrad(const WgradLaunch& L, cudaStream_t s) {
    using W = Wg<TAPS>;
    WgArgs a{};
    a.cin = L.cin; a.cout = L.cout;
    a.n = L.n; a.d = L.d; a.h = L.h; a.w = L.w;
    a.tiles_w = ceil_div(L.w, TW);
    a.tiles_h = ceil_div(L.h, TH);
    a.tiles_d = ceil_div(L.d, W::PD);
    const long long tiles = (long long)a.tiles_w * a.tiles_h * a.tiles_d * L.n;
    if (tiles >= (1ll << 31) || (long long)L.n * L.d >= (1ll << 31) - 1) return FSIM_E_INVALID;
    a.tiles = (int)tiles;
    a.nchunk = ceil_div(L.cin, W::OCT * 8);
    a.nparts = L.cout / NT;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return FSIM_E_CUDA;
    // one wave: a CTA keeps its accumulators over all its tiles and adds them once
    const int groups = a.nchunk * a.nparts;
    a.ksplit = sms / groups > 0 ? sms / groups : 1;
    if (a.ksplit > a.tiles) a.ksplit = a.tiles;
    // Drain depth (8 MMAs per step, a plane or a pair): an eighth of the CTA's steps or
    // less, 1 to 8.  Draining after every plane cost the MMAs a third of their rate (8 x
    // 64^3, 16 -> 16: 326 us against 230), and this stays below the depth at which the
    // sums were as exact as with the kernel before (all of a quarter as many voxels).
    constexpr int ZP = wgrad_zp<TAPS, NT>;
    const int steps = ceil_div(a.tiles, a.ksplit) * (W::PD / ZP) / (TAPS == 1 ? 2 : 1);
    a.interval = 1;
    while (a.interval < 8 && 2 * a.interval * 10 <= steps) a.interval *= 2;
    a.stage_bytes = W::X_BYTES + W::PD * (NT / 8) * W::G_OCT;
    a.ncols = tmem_cols(TAPS == 27 ? W::ACC * ZP * NT : 2 * NT);
    a.dw = L.dw;
    a.err = L.err;
    // the unused M groups of the last planes read past the X box, into the stage's G box
    if ((W::PD - 1) * W::X_PLANE + 16 * W::X_OCT > a.stage_bytes) return FSIM_E_INVALID;
    int smem = 2 * a.stage_bytes + 128;
    if (smem > SMEM_LIMIT) return FSIM_E_INVALID;
    if (smem < SMEM_LIMIT / 2 + 1024) smem = SMEM_LIMIT / 2 + 1024;  // one CTA per SM (TMEM)
    if (set_smem_limit((const void*)k_conv_wgrad<TAPS, NT>, SMEM_LIMIT) != cudaSuccess) return FSIM_E_CUDA;
    launch_dep(k_conv_wgrad<TAPS, NT>, (unsigned)(groups * a.ksplit), WG_THREADS, smem, s, a, *L.mx, *L.mg);
    return cudaGetLastError() == cudaSuccess ? FSIM_OK : FSIM_E_CUDA;
}

int launch_conv_wgrad(const WgradLaunch& L, cudaStream_t s) {
    if ((L.taps != 27 && L.taps != 1) || L.cin % 16 || L.cout % 16 || L.cin <= 0 || L.cout <= 0 || L.cout > 64)
        return FSIM_E_INVALID;
    if ((long long)L.n * L.d * L.h * L.w <= 0) return FSIM_OK;
    const int nt = wgrad_nt(L.taps, L.cout);
    if (L.taps == 27) return nt == 32 ? launch_wgrad<27, 32>(L, s) : launch_wgrad<27, 16>(L, s);
    switch (nt) {
        case 16: return launch_wgrad<1, 16>(L, s);
        case 32: return launch_wgrad<1, 32>(L, s);
        case 48: return launch_wgrad<1, 48>(L, s);
        default: return launch_wgrad<1, 64>(L, s);
    }
}
