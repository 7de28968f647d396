// k_render.cu -- headless screen-space fluid renderer (include/fsim_render.h).
//
// The passes of FluidSurfaceGfx::render (fluidSurfaceGfx.cpp:81-204) as CUDA
// kernels over device images (row 0 at the bottom, as OpenGL's window):
//   1. sprite depth splat of the surface particles (particle_sprites.vs +
//      particle_sprites_depth.fs): one thread per particle walks the pixels of
//      its billboard, finds the sprite coordinate of each pixel centre by
//      intersecting the pixel's eye ray with the billboard plane (what
//      perspective-correct interpolation of texCoord gives), and keeps the
//      nearest sphere depth with an atomicMin on the depth bits;
//   2. separable Gaussian (gaussian.fs) or bilateral (bilateral.fs) smoothing,
//      x then y, one thread per pixel;
//   3. spray particles (density below the threshold) splatted onto the
//      smoothed depth;
//   4. additive thickness splat (particle_sprites_thickness.fs) depth-tested
//      against the scene -- computed by passes 1 and 3 from the same fragments,
//      which cover every particle once -- then its separable blur
//      (gaussian_thickness.fs);
//   5. normals from the smoothed depth (normal_depth.fs);
//   6. Blinn-Phong shading with Perlin surface noise and thickness
//      transparency, blended over the background (shadedDepth.fs).
// All arithmetic is FP32 like the shaders; this file is compiled without FMA
// contraction so that the C restatement in oracle/ rounds the same way.
#include <cmath>
#include <cstring>
#include <string>

#include "../../include/fsim_render.h"
#include "fsim_common.cuh"

struct fsim_renderer {
    int W = 0, H = 0;
    int sms = 1;
    cudaStream_t own = nullptr;
    float* raw = nullptr;     // sprite depth (before smoothing)
    float* depth = nullptr;   // smoothed depth + spray
    float* tmp = nullptr;     // blur scratch
    float* thick = nullptr;   // thickness
    float* ttmp = nullptr;    // thickness blur scratch
    float4* nd = nullptr;     // normal + depth
    float4* color = nullptr;  // composited frame
    float* tab = nullptr;     // the blurs' weights, then the eye rays by axis
    fsim_particle_gfx* parts = nullptr;  // staging for host particles / fsim_render_ctx
    long long parts_cap = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaStream_t last = nullptr;
    int launches = 0;
    bool timed = false;
    std::string err;
};

namespace {

struct Mat4 {
    float m[16];  // column-major: m[c * 4 + r]
};

struct Cam {
    Mat4 view, view_inv, proj, proj_inv;
    float pos[4];
};

__device__ __forceinline__ void mul4(const Mat4& M, const float (&v)[4], float (&o)[4]) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
        float s = M.m[r] * v[0];
        s = s + M.m[4 + r] * v[1];
        s = s + M.m[8 + r] * v[2];
        s = s + M.m[12 + r] * v[3];
        o[r] = s;
    }
}

__device__ __forceinline__ float dot3(const float* a, const float* b) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

__device__ __forceinline__ void cross3(const float* a, const float* b, float* o) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

// a / b with y = 1 / b rounded: one Newton correction of a y (Markstein, IBM J. Res.
// Develop. 34, 1990), for quotients far from overflow and underflow
__device__ __forceinline__ float div_by(float a, float b, float y) {
    const float q = a * y;
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// GLSL normalize; a zero vector stays zero (GLSL leaves it undefined)
__device__ __forceinline__ void normalize3(float* v) {
    const float l = sqrtf(dot3(v, v));
    if (l > 1e-15f && l < 1e15f) {
        const float y = 1.f / l;
        v[0] = div_by(v[0], l, y);
        v[1] = div_by(v[1], l, y);
        v[2] = div_by(v[2], l, y);
    } else if (l > 0.f) {
        v[0] = v[0] / l;
        v[1] = v[1] / l;
        v[2] = v[2] / l;
    }
}

// uvToEye: window (texCoord, depth) -> eye-space position
__device__ __forceinline__ void uv_to_eye(const Cam& c, float u, float v, float d, float* e) {
    const float ndc[4] = {u * 2.f - 1.f, v * 2.f - 1.f, d * 2.f - 1.f, 1.f};
    float o[4];
    mul4(c.proj_inv, ndc, o);
    e[0] = o[0] / o[3];
    e[1] = o[1] / o[3];
    e[2] = o[2] / o[3];
}

// ---- 1, 3, 4: sprite splats -------------------------------------------------
// The billboard of particle_sprites.vs: z = normalize(eye position),
// x = normalize(cross((0,1,0), z)), y = normalize(cross(z, x)); the FlipSquare's
// corners (+-0.5, +-0.5) scaled by 2r, texCoord = (px + 0.5, 0.5 - py).
struct Sprite {
    float c[3], xa[3], ya[3], za[3];
    float d2, d2_inv;    // diameter
    int x0, x1, y0, y1;  // pixel range (inclusive)
};

__device__ __forceinline__ bool make_sprite(const Cam& cam, const float* pw, float r, int W, int H, Sprite& s) {
    s.d2 = r * 2.f;
    s.d2_inv = 1.f / s.d2;
    const float p4[4] = {pw[0], pw[1], pw[2], 1.f};
    float e[4];
    mul4(cam.view, p4, e);
    s.c[0] = e[0]; s.c[1] = e[1]; s.c[2] = e[2];
    s.za[0] = e[0]; s.za[1] = e[1]; s.za[2] = e[2];
    normalize3(s.za);
    const float up[3] = {0.f, 1.f, 0.f};
    cross3(up, s.za, s.xa);
    normalize3(s.xa);
    cross3(s.za, s.xa, s.ya);
    normalize3(s.ya);
    // projected corners -> pixel-centre range; a sprite reaching behind the eye is skipped
    float xmin = 1e30f, xmax = -1e30f, ymin = 1e30f, ymax = -1e30f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float sx = (k & 1) ? 0.5f : -0.5f, sy = (k & 2) ? 0.5f : -0.5f;
        float q[4];
#pragma unroll
        for (int a = 0; a < 3; a++) q[a] = s.c[a] + (s.xa[a] * sx + s.ya[a] * sy) * (r * 2.f);
        q[3] = 1.f;
        float cl[4];
        mul4(cam.proj, q, cl);
        if (!(cl[3] > 0.f)) return false;
        const float wx = (cl[0] / cl[3] * 0.5f + 0.5f) * (float)W, wy = (cl[1] / cl[3] * 0.5f + 0.5f) * (float)H;
        xmin = fminf(xmin, wx); xmax = fmaxf(xmax, wx);
        ymin = fminf(ymin, wy); ymax = fmaxf(ymax, wy);
    }
    // pixel i covers centre i + 0.5 (bounds clamped before the integer conversion)
    xmin = fmaxf(xmin, -1.f); ymin = fmaxf(ymin, -1.f);
    xmax = fminf(xmax, (float)W + 1.f); ymax = fminf(ymax, (float)H + 1.f);
    s.x0 = max((int)ceilf(xmin - 0.5f), 0);
    s.x1 = min((int)floorf(xmax - 0.5f), W - 1);
    s.y0 = max((int)ceilf(ymin - 0.5f), 0);
    s.y1 = min((int)floorf(ymax - 0.5f), H - 1);
    return s.x0 <= s.x1 && s.y0 <= s.y1;
}

// Eye ray of pixel (i, j): the eye-space point at its centre on the near plane.
__device__ __forceinline__ void eye_ray(const Cam& cam, int W, int H, int i, int j, float* d) {
    const float nd4[4] = {((float)i + 0.5f) / (float)W * 2.f - 1.f, ((float)j + 0.5f) / (float)H * 2.f - 1.f, -1.f,
                          1.f};
    float o[4];
    mul4(cam.proj_inv, nd4, o);
    d[0] = o[0] / o[3];
    d[1] = o[1] / o[3];
    d[2] = o[2] / o[3];
}
// Under a projection whose inverse keeps x and y apart (any but a sheared or rotated one)
// a ray's x depends on the column alone, its y on the row, and its z is the same for all:
// W + H + 1 numbers, tabulated once a frame (k_tables), which stay in L1.  The zero products
// left out change no sum.  Unprojecting the pixel for every fragment is 28 operations and
// five divisions of ~200; a table of all rays was 16 bytes written per pixel and read per
// fragment (2M sprites at 1000 x 1000: 436 us a frame with it, 366 now; 1000 small ones at
// 3840 x 2160: 382 and 330).
inline bool rays_by_axis(const Cam& cam) {
    const float* m = cam.proj_inv.m;
    return m[1] == 0.f && m[2] == 0.f && m[3] == 0.f && m[4] == 0.f && m[6] == 0.f && m[7] == 0.f;
}

// Sprite coordinate of the pixel with eye ray d: false outside the quad.  On return P is
// the eye-space point of the billboard plane under the pixel centre.
__device__ __forceinline__ bool sprite_hit(const float* d, const Sprite& s, float& px, float& py, float* P) {
    const float den = dot3(d, s.za);
    if (!(den > 0.f)) return false;
    const float t = dot3(s.c, s.za) / den;
    P[0] = d[0] * t; P[1] = d[1] * t; P[2] = d[2] * t;
    const float q[3] = {P[0] - s.c[0], P[1] - s.c[1], P[2] - s.c[2]};
    px = div_by(dot3(q, s.xa), s.d2, s.d2_inv);
    py = div_by(dot3(q, s.ya), s.d2, s.d2_inv);
    return fabsf(px) <= 0.5f && fabsf(py) <= 0.5f;
}

__device__ __forceinline__ float window_depth(const Cam& cam, const float* p, bool& inside) {
    const float q[4] = {p[0], p[1], p[2], 1.f};
    float cl[4];
    mul4(cam.proj, q, cl);
    const float z = cl[2] / cl[3];
    inside = z >= -1.f && z <= 1.f;  // near / far clipping
    return z * 0.5f + 0.5f;
}

// With `thick` set, a fragment also adds its thickness
// (particle_sprites_thickness.fs: sqrt(1 - r2) * r, GL_ONE + GL_ONE blending),
// depth-tested GL_LESS against the scene depth at the billboard plane and not
// against the fluid depth, so one pass per particle serves both splats (the
// surface and the spray passes together cover every particle once).
//
// Bound by arithmetic without contraction (IEEE divisions and square roots), so work
// whose outcome is known is left out.  plain_proj: the projection's depth depends on the
// eye depth alone and falls with it (any perspective).  Then no point of the sphere is
// nearer than its front, and a fragment behind the depth already there (most, many
// particles deep in the fluid) only adds its thickness; and between the near and the far
// plane every fragment passes the clip test and, without a scene, the depth test.  The
// margins cover the rounding of the depths, also where near and far are close and a depth
// (a |z| - b) / |z| is the difference of large products: the numerator is rounded
// monotonically in z, so two depths are out of order by 2^-22 at most, whatever a is; and a
// point of the billboard plane is nearer to the sprite's centre along z than r by more than
// its rounding unless it is seen at a right angle.
template <bool AXES>
__device__ __forceinline__ void splat(const float* pos, const Cam& cam, float r, int W, int H, const float* ray,
                                      int plain_proj, unsigned* depth_bits, const float* scene, float* thick) {
    Sprite s;
    if (!make_sprite(cam, pos, r, W, H, s)) return;
    float front = -1.f;  // no depth of the sphere is below it
    bool deep = false;   // every fragment lies between the near and the far plane
    if (plain_proj && s.c[2] + 1.001f * r < 0.f) {
        const float f[3] = {0.f, 0.f, s.c[2] + 1.001f * r}, b[3] = {0.f, 0.f, s.c[2] - 1.001f * r};
        bool in;
        const float zf = window_depth(cam, f, in), zb = window_depth(cam, b, in);
        if (zf == zf) front = zf - 4e-6f;
        deep = front > 1e-5f && zb < 1.f - 1e-5f;
    }
    float d[3];  // eye ray
    if (AXES) d[2] = ray[W + H];
    for (int j = s.y0; j <= s.y1; j++) {
        if (AXES) d[1] = ray[W + j];
        for (int i = s.x0; i <= s.x1; i++) {
            const int pix = j * W + i;
            float px, py, P[3];
            if (AXES) d[0] = ray[i];
            else eye_ray(cam, W, H, i, j, d);
            if (!sprite_hit(d, s, px, py, P)) continue;
            // particle_sprites_depth.fs
            const float nx = px * 2.f, ny = -py * 2.f;  // texCoord * 2 - 1
            const float r2 = nx * nx + ny * ny;
            if (r2 > 1.f) continue;
            bool lit = thick != nullptr;
            if (!deep || (scene && thick)) {
                bool inside;
                const float zq = window_depth(cam, P, inside);
                if (!inside) continue;
                lit = lit && zq < (scene ? scene[pix] : 1.f);
            }
            const float sq = sqrtf(1.f - r2);
            if (lit) atomicAdd(&thick[pix], sq * r);
            // (an older depth from L1 is larger: it only costs work)
            if (front > __uint_as_float(depth_bits[pix])) continue;
            float nrm[3];
#pragma unroll
            for (int a = 0; a < 3; a++) nrm[a] = s.xa[a] * nx + s.ya[a] * ny + s.za[a] * -sq;
            normalize3(nrm);
            float pp[3];
#pragma unroll
            for (int a = 0; a < 3; a++) pp[a] = s.c[a] + nrm[a] * r;
            bool in2;
            float z = window_depth(cam, pp, in2);
            z = fminf(fmaxf(z, 0.f), 1.f);  // gl_FragDepth is clamped to the depth range
            atomicMin(&depth_bits[pix], __float_as_uint(z));  // z >= 0: bits order as floats
        }
    }
}

// which: 0 all particles, 1 surface (density >= threshold), 2 spray (below).  The spray is
// a few particles of many: a block gathers the ones among `gather` before it splats them
// (with one thread per particle 3.4 of 32 lanes worked).  1000 x 1000 pixels, 8M
// particles: surface 629 us and spray 130 before, now 405 and 53.
constexpr int SPLAT_GATHER = 2048;
// A block's spray is splatted by its 256 threads in turn, so where a frame has little else
// a wide gather leaves the chip idle (2048 sprites, all spray, 1000 x 1000: one block and
// 3570 us a frame, eight of 256 618): eight blocks per SM come first, then wider ones.
static int splat_gather(long long n, int sms) {
    const long long per = (n + 8ll * sms - 1) / (8ll * sms), g = (per + 255) / 256 * 256;
    return (int)(g < 256 ? 256 : g > SPLAT_GATHER ? SPLAT_GATHER : g);
}
template <bool AXES, int MINB>
__global__ void __launch_bounds__(256, MINB) k_splat_depth(const fsim_particle_gfx* parts, long long n, int which, float thr,
                                                     Cam cam, float r, int W, int H, const float* ray, int plain_proj,
                                                     unsigned* depth_bits, const float* scene, float* thick, int gather) {
    pdl_enter();
    if (which != 2) {
        const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        if (k >= n) return;
        const fsim_particle_gfx pg = parts[k];
        if (which == 1 && pg.density < thr) return;
        splat<AXES>(pg.pos, cam, r, W, H, ray, plain_proj, depth_bits, scene, thick);
        return;
    }
    __shared__ int list[SPLAT_GATHER], count;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    const long long k0 = (long long)blockIdx.x * gather;
    const int m = (int)min((long long)gather, n - k0);
    for (int i = threadIdx.x; i < m; i += blockDim.x)
        if (parts[k0 + i].density < thr) list[atomicAdd(&count, 1)] = i;
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += blockDim.x)
        splat<AXES>(parts[k0 + list[i]].pos, cam, r, W, H, ray, plain_proj, depth_bits, scene, thick);
}

// The blurs' weights depend on the tap and the pixel's radius alone (26 Gaussian radii, and
// the bilateral filter's 36 taps): one table a frame, with the formulas of the shaders.
constexpr int BLUR_MAX_R = 25, BLUR_BI_R = 35;
constexpr int BLUR_GAUSS = (BLUR_MAX_R + 1) * (BLUR_MAX_R + 1), BLUR_TAB = BLUR_GAUSS + BLUR_BI_R + 1;
__device__ __forceinline__ float blur_weight(int q, float blur_scale) {
    if (q >= BLUR_GAUSS) {
        const float rr = (float)(q - BLUR_GAUSS) * blur_scale;
        return expf(-rr * rr);
    }
    const int R = q / (BLUR_MAX_R + 1), p = q % (BLUR_MAX_R + 1);
    if (R < 1 || p > R) return 0.f;
    const float sd = (float)(2 * R) / 6.f;
    const float sd2 = sd * sd;
    return expf((float)(-p * p) / sd2 * 0.5f);
}

// what depends on the frame's parameters alone: the blurs' weights and the rays by axis
__global__ void k_tables(Cam cam, int W, int H, float blur_scale, float* tab) {
    pdl_enter();
    const int q = blockIdx.x * blockDim.x + threadIdx.x, e = q - BLUR_TAB;  // e: column, row, or the rays' z
    if (e > W + H) return;
    float d[3];
    if (e >= 0) eye_ray(cam, W, H, e < W ? e : 0, e < W ? 0 : e - W, d);
    tab[q] = e < 0 ? blur_weight(q, blur_scale) : e < W ? d[0] : e < W + H ? d[1] : d[2];
}

__global__ void k_clear(float* depth, float* thick, long long n) {
    pdl_enter();
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    depth[k] = 1.f;
    thick[k] = 0.f;
}

// ---- 2, 4: separable blurs -----------------------------------------------------
// Kernel extent from the world-space smoothing size projected at the pixel
// (gaussian.fs / bilateral.fs / gaussian_thickness.fs).
__device__ __forceinline__ float screen_extent(const Cam& cam, const float* eye, float size, int axis, float u,
                                               float v) {
    float q[4] = {eye[0], eye[1], eye[2], 1.f};
    q[axis] = q[axis] + size * 0.5f;
    float o[4];
    mul4(cam.proj, q, o);
    return axis == 0 ? o[0] / o[3] * 0.5f + 0.5f - u : o[1] / o[3] * 0.5f + 0.5f - v;
}

// mode 0: Gaussian depth, 1: bilateral depth, 2: Gaussian thickness (src = thickness, dsrc = depth)
__device__ __forceinline__ void blur_pixel(int mode, int axis, const float* src, const float* dsrc, float* dst, int W,
                                           int H, const Cam& cam, float size, float falloff, const float* weights,
                                           int id, float cur) {
    const int x = id % W, y = id / W;
    const float u = ((float)x + 0.5f) / (float)W, v = ((float)y + 0.5f) / (float)H;
    float eye[3];
    uv_to_eye(cam, u, v, cur, eye);
    const int tex = axis == 0 ? W : H, at = axis == 0 ? x : y, step = axis == 0 ? 1 : W;
    // texel of tap p, clamped to the edge
    auto tap = [&](int p) { return src[id + (min(max(at + p, 0), tex - 1) - at) * step]; };
    const float ext = screen_extent(cam, eye, size, axis, u, v);
    float acc = 0.f, wsum = 0.f;
    if (mode == 1) {
        int R = (int)(ext * (float)tex);
        R = R > 35 ? 35 : (R < 1 ? 1 : R);
        for (int p = -R; p <= R; p++) {
            const float s = tap(p);
            if (s < 1.f) {
                const float w = weights[p < 0 ? -p : p];
                const float r2 = (s - cur) * falloff;
                const float g = expf(-r2 * r2);
                acc = acc + s * w * g;
                wsum = wsum + w * g;
            }
        }
        dst[id] = wsum == 0.f ? 1.f : acc / wsum;
        return;
    }
    int ks = (int)(ext * (float)tex) * 2 + 1;
    ks = ks > 51 ? 51 : (ks < 3 ? 3 : ks);
    const int R = ks / 2;
    const float* wr = weights + R * (BLUR_MAX_R + 1);
    auto add = [&](float s, float w) {
        if (mode == 2 || s < 1.f) {
            wsum = wsum + w;
            acc = acc + s * w;
        }
    };
    if (at >= R && at + R < tex) {  // no tap is clamped
        const float* q = src + id - R * step;
        for (int p = R; p > 0; p--, q += step) add(*q, wr[p]);
        for (int p = 0; p <= R; p++, q += step) add(*q, wr[p]);
    } else {
        for (int p = -R; p <= R; p++) add(tap(p), wr[p < 0 ? -p : p]);
    }
    dst[id] = acc / wsum;
}

// Background pixels leave before anything else (the depth is cleared there, the value
// stays), and no block prepares anything: with the table computed by every block of every
// pass (~350 exponentials and divisions), a frame of 3840 x 2160 that is nearly all
// background took 578 us; copying it to shared memory is no faster than reading it from
// L1.  DEP: launched as a dependent kernel.  A block's wait for the kernel before costs what
// a background block does, so a frame of many waves of blocks takes ordinary launches
// (3840 x 2160: 330 us with dependent ones, now 273).
template <bool DEP>
__global__ void k_blur(int mode, int axis, const float* src, const float* dsrc, float* dst, int W, int H, Cam cam,
                       float size, float falloff, const float* weights) {
    if (DEP) pdl_enter();
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= W * H) return;
    const float cur = dsrc[id];
    if (cur == 1.f) {
        dst[id] = mode == 2 ? 0.f : 1.f;
        return;
    }
    blur_pixel(mode, axis, src, dsrc, dst, W, H, cam, size, falloff, weights + (mode == 1 ? BLUR_GAUSS : 0), id, cur);
}

// ---- 5: normals (normal_depth.fs) ---------------------------------------------
__device__ __forceinline__ void eye_at(const Cam& cam, const float* depth, int W, int H, int x, int y, float* e) {
    const int cx = min(max(x, 0), W - 1), cy = min(max(y, 0), H - 1);
    // texCoord + texel offset, sampled with GL_NEAREST and CLAMP_TO_EDGE: the
    // coordinate is the unclamped one, the value the clamped texel's
    const float u = ((float)x + 0.5f) / (float)W, v = ((float)y + 0.5f) / (float)H;
    uv_to_eye(cam, u, v, depth[(long long)cy * W + cx], e);
}

__global__ void k_normals(const float* depth, float4* nd, int W, int H, Cam cam) {
    pdl_enter();
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)W * H) return;
    const int x = (int)(id % W), y = (int)(id / W);
    const float d = depth[id];
    if (d == 1.f) {
        nd[id] = make_float4(0.f, 0.f, 0.f, 1.f);
        return;
    }
    float p[3], a[3], b[3], ddx[3], ddx2[3], ddy[3], ddy2[3];
    eye_at(cam, depth, W, H, x, y, p);
    eye_at(cam, depth, W, H, x + 1, y, a);
    eye_at(cam, depth, W, H, x - 1, y, b);
#pragma unroll
    for (int k = 0; k < 3; k++) { ddx[k] = a[k] - p[k]; ddx2[k] = p[k] - b[k]; }
    if (fabsf(ddx[2]) > fabsf(ddx2[2])) { ddx[0] = ddx2[0]; ddx[1] = ddx2[1]; ddx[2] = ddx2[2]; }
    eye_at(cam, depth, W, H, x, y + 1, a);
    eye_at(cam, depth, W, H, x, y - 1, b);
#pragma unroll
    for (int k = 0; k < 3; k++) { ddy[k] = a[k] - p[k]; ddy2[k] = p[k] - b[k]; }
    if (fabsf(ddy2[2]) < fabsf(ddy[2])) { ddy[0] = ddy2[0]; ddy[1] = ddy2[1]; ddy[2] = ddy2[2]; }
    float n[3];
    cross3(ddx, ddy, n);
    normalize3(n);
    const float n4[4] = {n[0], n[1], n[2], 0.f};
    float w[4];
    mul4(cam.view_inv, n4, w);
    nd[id] = make_float4(w[0], w[1], w[2], d);
}

// ---- 6: shading (shadedDepth.fs) ------------------------------------------------
// Classic 3D Perlin noise in the form of Gustavson's shader: lattice hashes by
// the permutation polynomial (34 x + 10) x mod 289, gradients on the surface
// of an octahedron from the hash, quintic fade, scaled by 2.2.
__device__ __forceinline__ float mod289(float x) { return x - floorf(x * (1.f / 289.f)) * 289.f; }
__device__ __forceinline__ float permute(float x) { return mod289((x * 34.f + 10.f) * x); }
__device__ __forceinline__ float fractf(float x) { return x - floorf(x); }
__device__ __forceinline__ float fade(float t) { return t * t * t * (t * (t * 6.f - 15.f) + 10.f); }
__device__ __forceinline__ float mixf(float a, float b, float t) { return a * (1.f - t) + b * t; }

__device__ float perlin(float X, float Y, float Z) {
    const float i0[3] = {mod289(floorf(X)), mod289(floorf(Y)), mod289(floorf(Z))};
    const float i1[3] = {mod289(floorf(X) + 1.f), mod289(floorf(Y) + 1.f), mod289(floorf(Z) + 1.f)};
    const float f0[3] = {fractf(X), fractf(Y), fractf(Z)};
    const float f1[3] = {f0[0] - 1.f, f0[1] - 1.f, f0[2] - 1.f};
    float n[2][4];  // [z corner][xy corner: (0,0) (1,0) (0,1) (1,1)]
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int cx = c & 1, cy = c >> 1;
        const float hxy = permute(permute(cx ? i1[0] : i0[0]) + (cy ? i1[1] : i0[1]));
#pragma unroll
        for (int cz = 0; cz < 2; cz++) {
            const float h = permute(hxy + (cz ? i1[2] : i0[2]));
            float gx = h * (1.f / 7.f);
            float gy = fractf(floorf(gx) * (1.f / 7.f)) - 0.5f;
            gx = fractf(gx);
            const float gz = 0.5f - fabsf(gx) - fabsf(gy);
            const float sz = gz <= 0.f ? 1.f : 0.f;  // step(gz, 0)
            gx = gx - sz * ((gx < 0.f ? 0.f : 1.f) - 0.5f);
            gy = gy - sz * ((gy < 0.f ? 0.f : 1.f) - 0.5f);
            const float norm = 1.79284291400159f - 0.85373472095314f * (gx * gx + gy * gy + gz * gz);
            n[cz][c] = (gx * norm) * (cx ? f1[0] : f0[0]) + (gy * norm) * (cy ? f1[1] : f0[1]) +
                       (gz * norm) * (cz ? f1[2] : f0[2]);
        }
    }
    const float fx = fade(f0[0]), fy = fade(f0[1]), fz = fade(f0[2]);
    float nz[4];
#pragma unroll
    for (int c = 0; c < 4; c++) nz[c] = mixf(n[0][c], n[1][c], fz);
    const float ny0 = mixf(nz[0], nz[2], fy), ny1 = mixf(nz[1], nz[3], fy);
    return 2.2f * mixf(ny0, ny1, fx);
}

struct ShadeArgs {
    Cam cam;
    int W, H;
    const float4* nd;
    const float* thick;
    const float* scene;
    float4* color;
    float diffuse[4], specular[3], shininess;
    int transparency_enabled;
    float transparency;
    int noise_enabled;
    float noise_scale, noise_strength, noise_offset;
    int nl;
    fsim_light lights[FSIM_RENDER_MAX_LIGHTS];
    float bg[4];
};

__device__ __forceinline__ void world_at(const ShadeArgs& a, int x, int y, float* w, float* nrm) {
    const int cx = min(max(x, 0), a.W - 1), cy = min(max(y, 0), a.H - 1);
    const float4 t = a.nd[(long long)cy * a.W + cx];
    const float u = ((float)x + 0.5f) / (float)a.W, v = ((float)y + 0.5f) / (float)a.H;
    float e[3];
    uv_to_eye(a.cam, u, v, t.w, e);
    const float e4[4] = {e[0], e[1], e[2], 1.f};
    float o[4];
    mul4(a.cam.view_inv, e4, o);
    w[0] = o[0]; w[1] = o[1]; w[2] = o[2];
    nrm[0] = t.x; nrm[1] = t.y; nrm[2] = t.z;
}

// getNoiseOffsetWorldSpacePos
__device__ __forceinline__ void noisy_pos(const ShadeArgs& a, int x, int y, float* out) {
    float w[3], n[3];
    world_at(a, x, y, w, n);
    const float px = w[0] * a.noise_scale, py = w[1] * a.noise_scale, pz = w[2] * a.noise_scale;
    const float noise =
        perlin(px + a.noise_offset, py, pz) + perlin(-px + a.noise_offset, py + a.noise_offset, pz);
#pragma unroll
    for (int k = 0; k < 3; k++) out[k] = w[k] + n[k] * noise;
}

__device__ void shade_light(const float* wp, const float* nrm_in, const float* view, const fsim_light& L,
                            const float* mat, const float* spec, float shininess, float* acc) {
    float f2l[3];
#pragma unroll
    for (int k = 0; k < 3; k++) f2l[k] = L.position[k] - wp[k] * L.position[3];
    float ld[3] = {f2l[0], f2l[1], f2l[2]};
    normalize3(ld);
    float n[3] = {nrm_in[0], nrm_in[1], nrm_in[2]};
    if (dot3(n, view) < 0.f) { n[0] = -n[0]; n[1] = -n[1]; n[2] = -n[2]; }
    const float lc = dot3(ld, n);
    if (lc < 0.f) return;
    float d2 = sqrtf(dot3(f2l, f2l));
    d2 = d2 * d2;
    float hw[3] = {view[0] + ld[0], view[1] + ld[1], view[2] + ld[2]};
    normalize3(hw);
    float shine = dot3(hw, n);
    if (shine < 0.f) shine = 0.f;
    const float sp = powf(shine, shininess);
#pragma unroll
    for (int k = 0; k < 3; k++) acc[k] = acc[k] + L.power_density[k] * (mat[k] * lc + spec[k] * sp) / d2;
}

// Blocks of 32 x 8 pixels.  A pixel's noise normal needs the displaced positions of its
// four neighbours, which are the neighbours' own: the block evaluates each position (two
// noise values, ~400 operations each) once into shared memory, with a one-pixel rim, 1.3
// per pixel instead of 5 (91 us at 1000 x 1000, now 36).
constexpr int SHADE_X = 32, SHADE_Y = 8;
__global__ void __launch_bounds__(SHADE_X * SHADE_Y) k_shade(const ShadeArgs a) {
    pdl_enter();
    constexpr int PX = SHADE_X + 2, PY = SHADE_Y + 2;
    __shared__ float pos[3][PY * PX];
    const int tiles_x = (a.W + SHADE_X - 1) / SHADE_X;
    const int bx = (int)(blockIdx.x % tiles_x) * SHADE_X, by = (int)(blockIdx.x / tiles_x) * SHADE_Y;
    const int x = bx + (int)(threadIdx.x % SHADE_X), y = by + (int)(threadIdx.x / SHADE_X);
    const bool in = x < a.W && y < a.H;
    const long long id = (long long)y * a.W + x;
    const float4 t = in ? a.nd[id] : make_float4(0.f, 0.f, 0.f, 1.f);
    const float4 bg = make_float4(a.bg[0], a.bg[1], a.bg[2], a.bg[3]);
    const bool surface = in && !(t.w == 1.f || (a.scene && !(t.w < a.scene[id])));
    if (in && !surface) a.color[id] = bg;
    if (!__syncthreads_or(surface)) return;
    if (a.noise_enabled) {
        for (int q = threadIdx.x; q < PX * PY; q += SHADE_X * SHADE_Y) {
            float p[3];
            noisy_pos(a, bx - 1 + q % PX, by - 1 + q / PX, p);
#pragma unroll
            for (int k = 0; k < 3; k++) pos[k][q] = p[k];
        }
        __syncthreads();
    }
    if (!surface) return;
    float wp[3], n[3];
    world_at(a, x, y, wp, n);
    if (a.noise_enabled) {
        float p[3], q[3], ddx[3], ddx2[3], ddy[3], ddy2[3];
        const int at = (y - by + 1) * PX + x - bx + 1;
        auto read = [&](int o, float (&v)[3]) {
#pragma unroll
            for (int k = 0; k < 3; k++) v[k] = pos[k][at + o];
        };
        read(0, p);
        read(1, q);
#pragma unroll
        for (int k = 0; k < 3; k++) ddx[k] = q[k] - p[k];
        read(-1, q);
#pragma unroll
        for (int k = 0; k < 3; k++) ddx2[k] = p[k] - q[k];
        if (fabsf(ddx[2]) > fabsf(ddx2[2])) { ddx[0] = ddx2[0]; ddx[1] = ddx2[1]; ddx[2] = ddx2[2]; }
        read(PX, q);
#pragma unroll
        for (int k = 0; k < 3; k++) ddy[k] = q[k] - p[k];
        read(-PX, q);
#pragma unroll
        for (int k = 0; k < 3; k++) ddy2[k] = p[k] - q[k];
        if (fabsf(ddy2[2]) < fabsf(ddy[2])) { ddy[0] = ddy2[0]; ddy[1] = ddy2[1]; ddy[2] = ddy2[2]; }
        float nn[3];
        cross3(ddx, ddy, nn);
        normalize3(nn);
        const float s = a.noise_strength;
#pragma unroll
        for (int k = 0; k < 3; k++) n[k] = n[k] * (1.f - s) + nn[k] * s;
        normalize3(n);
    }
    float c[4] = {0.f, 0.f, 0.f, a.diffuse[3]};
    if (a.transparency_enabled) c[3] = expf(-a.transparency * a.thick[id]);
    float view[3] = {a.cam.pos[0] - wp[0], a.cam.pos[1] - wp[1], a.cam.pos[2] - wp[2]};
    normalize3(view);
    for (int l = 0; l < a.nl; l++) shade_light(wp, n, view, a.lights[l], a.diffuse, a.specular, a.shininess, c);
    if (a.transparency_enabled) {
        // glBlendFunc(GL_ONE_MINUS_SRC_ALPHA, GL_SRC_ALPHA) over the background
        const float al = c[3];
        a.color[id] = make_float4(c[0] * (1.f - al) + bg.x * al, c[1] * (1.f - al) + bg.y * al,
                                  c[2] * (1.f - al) + bg.z * al, c[3] * (1.f - al) + bg.w * al);
    } else {
        a.color[id] = make_float4(c[0], c[1], c[2], c[3]);
    }
}

// ---- host helpers ----------------------------------------------------------------
inline unsigned nblk(long long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

void to_cam(const fsim_camera& c, Cam& k) {
    std::memcpy(k.view.m, c.view, sizeof(k.view.m));
    std::memcpy(k.view_inv.m, c.view_inv, sizeof(k.view_inv.m));
    std::memcpy(k.proj.m, c.proj, sizeof(k.proj.m));
    std::memcpy(k.proj_inv.m, c.proj_inv, sizeof(k.proj_inv.m));
    std::memcpy(k.pos, c.position, sizeof(k.pos));
}

// general 4x4 inverse (cofactor expansion), column-major
bool invert4(const double* m, double* inv) {
    double t[16];
    t[0] = m[5] * m[10] * m[15] - m[5] * m[11] * m[14] - m[9] * m[6] * m[15] + m[9] * m[7] * m[14] +
           m[13] * m[6] * m[11] - m[13] * m[7] * m[10];
    t[4] = -m[4] * m[10] * m[15] + m[4] * m[11] * m[14] + m[8] * m[6] * m[15] - m[8] * m[7] * m[14] -
           m[12] * m[6] * m[11] + m[12] * m[7] * m[10];
    t[8] = m[4] * m[9] * m[15] - m[4] * m[11] * m[13] - m[8] * m[5] * m[15] + m[8] * m[7] * m[13] +
           m[12] * m[5] * m[11] - m[12] * m[7] * m[9];
    t[12] = -m[4] * m[9] * m[14] + m[4] * m[10] * m[13] + m[8] * m[5] * m[14] - m[8] * m[6] * m[13] -
            m[12] * m[5] * m[10] + m[12] * m[6] * m[9];
    t[1] = -m[1] * m[10] * m[15] + m[1] * m[11] * m[14] + m[9] * m[2] * m[15] - m[9] * m[3] * m[14] -
           m[13] * m[2] * m[11] + m[13] * m[3] * m[10];
    t[5] = m[0] * m[10] * m[15] - m[0] * m[11] * m[14] - m[8] * m[2] * m[15] + m[8] * m[3] * m[14] +
           m[12] * m[2] * m[11] - m[12] * m[3] * m[10];
    t[9] = -m[0] * m[9] * m[15] + m[0] * m[11] * m[13] + m[8] * m[1] * m[15] - m[8] * m[3] * m[13] -
           m[12] * m[1] * m[11] + m[12] * m[3] * m[9];
    t[13] = m[0] * m[9] * m[14] - m[0] * m[10] * m[13] - m[8] * m[1] * m[14] + m[8] * m[2] * m[13] +
            m[12] * m[1] * m[10] - m[12] * m[2] * m[9];
    t[2] = m[1] * m[6] * m[15] - m[1] * m[7] * m[14] - m[5] * m[2] * m[15] + m[5] * m[3] * m[14] +
           m[13] * m[2] * m[7] - m[13] * m[3] * m[6];
    t[6] = -m[0] * m[6] * m[15] + m[0] * m[7] * m[14] + m[4] * m[2] * m[15] - m[4] * m[3] * m[14] -
           m[12] * m[2] * m[7] + m[12] * m[3] * m[6];
    t[10] = m[0] * m[5] * m[15] - m[0] * m[7] * m[13] - m[4] * m[1] * m[15] + m[4] * m[3] * m[13] +
            m[12] * m[1] * m[7] - m[12] * m[3] * m[5];
    t[14] = -m[0] * m[5] * m[14] + m[0] * m[6] * m[13] + m[4] * m[1] * m[14] - m[4] * m[2] * m[13] -
            m[12] * m[1] * m[6] + m[12] * m[2] * m[5];
    t[3] = -m[1] * m[6] * m[11] + m[1] * m[7] * m[10] + m[5] * m[2] * m[11] - m[5] * m[3] * m[10] -
           m[9] * m[2] * m[7] + m[9] * m[3] * m[6];
    t[7] = m[0] * m[6] * m[11] - m[0] * m[7] * m[10] - m[4] * m[2] * m[11] + m[4] * m[3] * m[10] +
           m[8] * m[2] * m[7] - m[8] * m[3] * m[6];
    t[11] = -m[0] * m[5] * m[11] + m[0] * m[7] * m[9] + m[4] * m[1] * m[11] - m[4] * m[3] * m[9] -
            m[8] * m[1] * m[7] + m[8] * m[3] * m[5];
    t[15] = m[0] * m[5] * m[10] - m[0] * m[6] * m[9] - m[4] * m[1] * m[10] + m[4] * m[2] * m[9] +
            m[8] * m[1] * m[6] - m[8] * m[2] * m[5];
    const double det = m[0] * t[0] + m[1] * t[4] + m[2] * t[8] + m[3] * t[12];
    if (det == 0.0) return false;
    for (int i = 0; i < 16; i++) inv[i] = t[i] / det;
    return true;
}

int fail(fsim_renderer* r, int code, const std::string& msg) {
    if (r) r->err = msg;
    return code;
}

int ensure_parts(fsim_renderer* r, long long n) {
    if (n <= r->parts_cap) return FSIM_OK;
    cudaFree(r->parts);
    r->parts = nullptr;
    r->parts_cap = 0;
    const long long cap = n + n / 4 + 1024;
    if (cudaMalloc(&r->parts, (size_t)cap * sizeof(fsim_particle_gfx)) != cudaSuccess) {
        cudaGetLastError();
        return fail(r, FSIM_E_OOM, "particle staging buffer");
    }
    r->parts_cap = cap;
    return FSIM_OK;
}

}  // namespace

extern "C" {

void fsim_render_default_params(fsim_render_params* p) {
    if (!p) return;
    std::memset(p, 0, sizeof(*p));
    p->particle_radius = 1.f / 1024.f;
    p->particle_color[0] = 0.f; p->particle_color[1] = 0.4f; p->particle_color[2] = 0.95f;
    p->specular_color[0] = p->specular_color[1] = p->specular_color[2] = 1.2f;
    p->shininess = 80.f;
    p->bilateral_filter = 0;
    p->smoothing_size = 2.4f;
    p->blur_scale = 0.083f;
    p->blur_depth_falloff = 1100.f;
    p->spray_enabled = 1;
    p->spray_density_threshold = 1.2f;
    p->transparency_enabled = 1;
    p->transparency_blur_size = 2.4f;
    p->transparency = 1.334f;
    p->noise_enabled = 1;
    p->noise_scale = 0.956f;
    p->noise_strength = 0.123f;
    p->noise_offset = 0.f;
    const float lp[4][4] = {{50, 50, 50, 1}, {50, 50, -50, 1}, {-50, 50, -50, 1}, {-50, 50, 50, 1}};
    const float pd[4][3] = {{1000, 2000, 2000}, {2000, 1000, 2000}, {2000, 2000, 1000}, {2000, 2000, 2000}};
    p->num_lights = 4;
    for (int l = 0; l < 4; l++) {
        std::memcpy(p->lights[l].position, lp[l], sizeof(lp[l]));
        std::memcpy(p->lights[l].power_density, pd[l], sizeof(pd[l]));
    }
    p->background[0] = p->background[1] = p->background[2] = 0.f;
    p->background[3] = 1.f;
}

void fsim_render_camera(fsim_camera* cam, const double eye[3], double yaw_deg, double pitch_deg, double fov_deg,
                        double aspect, double z_near, double z_far) {
    if (!cam || !eye) return;
    const double kPi = 3.14159265358979323846;
    const double yaw = yaw_deg * kPi / 180.0, pitch = pitch_deg * kPi / 180.0;
    double f[3] = {std::cos(yaw) * std::cos(pitch), std::sin(pitch), std::sin(yaw) * std::cos(pitch)};
    auto norm = [](double* v) {
        const double l = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        v[0] /= l; v[1] /= l; v[2] /= l;
    };
    auto cross = [](const double* a, const double* b, double* o) {
        o[0] = a[1] * b[2] - a[2] * b[1];
        o[1] = a[2] * b[0] - a[0] * b[2];
        o[2] = a[0] * b[1] - a[1] * b[0];
    };
    norm(f);
    // Camera3D::updateViewMatrix: right = cross(front, +y), up = cross(right, front)
    const double yup[3] = {0, 1, 0};
    double right[3], up[3];
    cross(f, yup, right);
    norm(right);
    cross(right, f, up);
    norm(up);
    // lookAt(eye, eye + f, up), right-handed
    double s[3], u[3];
    cross(f, up, s);
    norm(s);
    cross(s, f, u);
    double V[16] = {0};
    V[0] = s[0]; V[4] = s[1]; V[8] = s[2];
    V[1] = u[0]; V[5] = u[1]; V[9] = u[2];
    V[2] = -f[0]; V[6] = -f[1]; V[10] = -f[2];
    V[12] = -(s[0] * eye[0] + s[1] * eye[1] + s[2] * eye[2]);
    V[13] = -(u[0] * eye[0] + u[1] * eye[1] + u[2] * eye[2]);
    V[14] = f[0] * eye[0] + f[1] * eye[1] + f[2] * eye[2];
    V[15] = 1;
    // perspective(fov, aspect, near, far), OpenGL clip depth [-1, 1]
    const double th = std::tan(fov_deg * kPi / 180.0 / 2.0);
    double P[16] = {0};
    P[0] = 1.0 / (aspect * th);
    P[5] = 1.0 / th;
    P[10] = -(z_far + z_near) / (z_far - z_near);
    P[11] = -1.0;
    P[14] = -(2.0 * z_far * z_near) / (z_far - z_near);
    double Vi[16], Pi[16];
    invert4(V, Vi);
    invert4(P, Pi);
    for (int i = 0; i < 16; i++) {
        cam->view[i] = (float)V[i];
        cam->view_inv[i] = (float)Vi[i];
        cam->proj[i] = (float)P[i];
        cam->proj_inv[i] = (float)Pi[i];
    }
    cam->position[0] = (float)eye[0];
    cam->position[1] = (float)eye[1];
    cam->position[2] = (float)eye[2];
    cam->position[3] = 1.f;
}

int fsim_render_create(int width, int height, fsim_renderer** out) {
    if (!out || width <= 0 || height <= 0 || (long long)width * height > (1ll << 28)) return FSIM_E_INVALID;
    *out = nullptr;
    fsim_renderer* r = new (std::nothrow) fsim_renderer();
    if (!r) return FSIM_E_OOM;
    r->W = width;
    r->H = height;
    const size_t np = (size_t)width * height;
    int dev = 0;
    bool ok = cudaGetDevice(&dev) == cudaSuccess &&
              cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
              cudaStreamCreateWithFlags(&r->own, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&r->raw, np * 4) == cudaSuccess && cudaMalloc(&r->depth, np * 4) == cudaSuccess &&
              cudaMalloc(&r->tmp, np * 4) == cudaSuccess && cudaMalloc(&r->thick, np * 4) == cudaSuccess &&
              cudaMalloc(&r->ttmp, np * 4) == cudaSuccess && cudaMalloc(&r->nd, np * 16) == cudaSuccess &&
              cudaMalloc(&r->color, np * 16) == cudaSuccess && cudaMalloc(&r->tab, ((size_t)BLUR_TAB + width + height + 1) * 4) == cudaSuccess && cudaEventCreate(&r->ev0) == cudaSuccess &&
              cudaEventCreate(&r->ev1) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        fsim_render_destroy(r);
        return FSIM_E_OOM;
    }
    *out = r;
    return FSIM_OK;
}

int fsim_render_destroy(fsim_renderer* r) {
    if (!r) return FSIM_OK;
    if (r->own) cudaStreamSynchronize(r->own);
    if (r->last) cudaStreamSynchronize(r->last);
    cudaFree(r->raw); cudaFree(r->depth); cudaFree(r->tmp); cudaFree(r->thick); cudaFree(r->ttmp);
    cudaFree(r->nd); cudaFree(r->color); cudaFree(r->tab); cudaFree(r->parts);
    if (r->ev0) cudaEventDestroy(r->ev0);
    if (r->ev1) cudaEventDestroy(r->ev1);
    if (r->own) cudaStreamDestroy(r->own);
    delete r;
    return FSIM_OK;
}

const char* fsim_render_last_error(fsim_renderer* r) { return r ? r->err.c_str() : "null renderer"; }

int fsim_render_frame(fsim_renderer* r, const fsim_particle_gfx* particles, int64_t n, int where,
                      const fsim_camera* cam, const fsim_render_params* prm, const float* scene_depth,
                      void* stream) {
    if (!r || !cam || !prm || n < 0 || (n > 0 && !particles)) return fail(r, FSIM_E_INVALID, "invalid argument");
    if (prm->num_lights < 0 || prm->num_lights > FSIM_RENDER_MAX_LIGHTS || !(prm->particle_radius > 0.f))
        return fail(r, FSIM_E_INVALID, "num_lights or particle_radius");
    cudaStream_t s = stream ? (cudaStream_t)stream : r->own;
    r->last = s;
    const fsim_particle_gfx* dp = particles;
    if (where == FSIM_HOST && n > 0) {
        int rc = ensure_parts(r, n);
        if (rc) return rc;
        if (cudaMemcpyAsync(r->parts, particles, (size_t)n * sizeof(fsim_particle_gfx), cudaMemcpyHostToDevice,
                            s) != cudaSuccess)
            return fail(r, FSIM_E_CUDA, "particle upload");
        dp = r->parts;
    }
    Cam k;
    to_cam(*cam, k);
    const int W = r->W, H = r->H;
    const long long np = (long long)W * H;
    const float rad = prm->particle_radius;
    int L = 0;
    cudaEventRecord(r->ev0, s);
    // 1. surface sprites into the cleared depth buffer, with their thickness
    //    (the thickness of all particles accumulates over passes 1 and 3)
    float* thick = prm->transparency_enabled ? r->thick : nullptr;
    const float* ray = r->tab + BLUR_TAB;
    // Many sprites hide their latency with resident blocks (32 registers and 200 bytes spilled:
    // 8M at 1000 x 1000 606 us a frame, 658 with 48 registers); a frame of at most four blocks
    // per SM has none to add and takes the registers (500 sprites of ~10,000 pixels 8850 -> 7980 us)
    const bool few = nblk(n) <= 4u * (unsigned)r->sms;
    auto* splat_depth = rays_by_axis(k) ? (few ? k_splat_depth<true, 4> : k_splat_depth<true, 8>)
                                        : (few ? k_splat_depth<false, 4> : k_splat_depth<false, 8>);
    const float* pm = k.proj.m;
    const int plain = pm[2] == 0.f && pm[6] == 0.f && pm[3] == 0.f && pm[7] == 0.f && pm[15] == 0.f && pm[11] < 0.f &&
                      pm[14] < 0.f;
    launch_dep(k_tables, nblk(BLUR_TAB + W + H + 1), 256, 0, s, k, W, H, prm->blur_scale, r->tab);
    launch_dep(k_clear, nblk(np), 256, 0, s, r->raw, r->thick, np);
    L += 2;
    if (n > 0) {
        launch_dep(splat_depth, nblk(n), 256, 0, s, dp, n, prm->spray_enabled ? 1 : 0, prm->spray_density_threshold, k, rad, W, H,
                   ray, plain, reinterpret_cast<unsigned*>(r->raw), scene_depth, thick, 0);
        L++;
    }
    // 2. smoothing, x into tmp then y into depth
    const int mode = prm->bilateral_filter ? 1 : 0;
    const bool many = np >= 8ll * 256 * 8 * r->sms;  // eight waves of eight blocks per SM
    auto blur = [&](int m, int axis, const float* src, const float* dsrc, float* dst, float size, float falloff) {
        if (many) k_blur<false><<<nblk(np), 256, 0, s>>>(m, axis, src, dsrc, dst, W, H, k, size, falloff, r->tab);
        else launch_dep(k_blur<true>, nblk(np), 256, 0, s, m, axis, src, dsrc, dst, W, H, k, size, falloff, r->tab);
        L++;
    };
    blur(mode, 0, r->raw, r->raw, r->tmp, prm->smoothing_size, prm->blur_depth_falloff);
    blur(mode, 1, r->tmp, r->tmp, r->depth, prm->smoothing_size, prm->blur_depth_falloff);
    // 3. spray on top of the smoothed surface
    if (prm->spray_enabled && n > 0) {
        const int gather = splat_gather(n, r->sms);
        launch_dep(splat_depth, nblk(n, gather), 256, 0, s, dp, n, 2, prm->spray_density_threshold, k, rad, W, H, ray, plain,
                   reinterpret_cast<unsigned*>(r->depth), scene_depth, thick, gather);
        L++;
    }
    // 4. thickness blurred x then y
    if (prm->transparency_enabled) {
        blur(2, 0, r->thick, r->depth, r->ttmp, prm->transparency_blur_size, 0.f);
        blur(2, 1, r->ttmp, r->depth, r->thick, prm->transparency_blur_size, 0.f);
    }
    // 5. normals
    launch_dep(k_normals, nblk(np), 256, 0, s, r->depth, r->nd, W, H, k);
    L++;
    // 6. shading and composite
    ShadeArgs a;
    a.cam = k;
    a.W = W;
    a.H = H;
    a.nd = r->nd;
    a.thick = r->thick;
    a.scene = scene_depth;
    a.color = r->color;
    for (int q = 0; q < 3; q++) {
        a.diffuse[q] = prm->particle_color[q];
        a.specular[q] = prm->specular_color[q];
    }
    a.diffuse[3] = 1.f;
    a.shininess = prm->shininess;
    a.transparency_enabled = prm->transparency_enabled;
    a.transparency = prm->transparency;
    a.noise_enabled = prm->noise_enabled;
    a.noise_scale = prm->noise_scale;
    a.noise_strength = prm->noise_strength;
    a.noise_offset = prm->noise_offset;
    a.nl = prm->num_lights;
    std::memcpy(a.lights, prm->lights, sizeof(a.lights));
    std::memcpy(a.bg, prm->background, sizeof(a.bg));
    launch_dep(k_shade, (unsigned)(((W + SHADE_X - 1) / SHADE_X) * ((H + SHADE_Y - 1) / SHADE_Y)), SHADE_X * SHADE_Y, 0, s, a);
    L++;
    cudaEventRecord(r->ev1, s);
    r->timed = true;
    r->launches = L;
    if (cudaGetLastError() != cudaSuccess) return fail(r, FSIM_E_CUDA, "render kernel launch failed");
    return FSIM_OK;
}

int fsim_render_read(fsim_renderer* r, int image, void* dst, int where) {
    if (!r || !dst) return FSIM_E_INVALID;
    const size_t np = (size_t)r->W * r->H;
    const void* src = nullptr;
    size_t bytes = np * 4;
    switch (image) {
        case FSIM_IMG_COLOR: src = r->color; bytes = np * 16; break;
        case FSIM_IMG_DEPTH: src = r->depth; break;
        case FSIM_IMG_THICKNESS: src = r->thick; break;
        case FSIM_IMG_NORMAL_DEPTH: src = r->nd; bytes = np * 16; break;
        case FSIM_IMG_RAW_DEPTH: src = r->raw; break;
        default: return fail(r, FSIM_E_INVALID, "unknown image");
    }
    cudaStream_t s = r->last ? r->last : r->own;
    if (cudaMemcpyAsync(dst, src, bytes, where == FSIM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice,
                        s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return fail(r, FSIM_E_CUDA, "image copy");
    return FSIM_OK;
}

int fsim_render_stats(fsim_renderer* r, float* ms, int* launches) {
    if (!r) return FSIM_E_INVALID;
    if (launches) *launches = r->launches;
    if (ms) {
        *ms = 0.f;
        if (r->timed) {
            if (cudaEventSynchronize(r->ev1) != cudaSuccess ||
                cudaEventElapsedTime(ms, r->ev0, r->ev1) != cudaSuccess) {
                cudaGetLastError();
                return fail(r, FSIM_E_CUDA, "frame timing");
            }
        }
    }
    return FSIM_OK;
}

int fsim_render_ctx(fsim_renderer* r, fsim_ctx* ctx, const fsim_camera* cam, const fsim_render_params* params,
                    const float* scene_depth) {
    if (!r || !ctx) return FSIM_E_INVALID;
    int64_t n = 0;
    int rc = fsim_num_particles(ctx, &n);
    if (rc) return fail(r, rc, "fsim_num_particles");
    if ((rc = ensure_parts(r, n))) return rc;
    int64_t got = 0;
    if (n > 0 && (rc = fsim_fill_gfx(ctx, r->parts, r->parts_cap, &got, FSIM_DEVICE)))
        return fail(r, rc, std::string("fsim_fill_gfx: ") + fsim_last_error(ctx));
    return fsim_render_frame(r, r->parts, got, FSIM_DEVICE, cam, params, scene_depth, fsim_stream(ctx));
}

}  // extern "C"
