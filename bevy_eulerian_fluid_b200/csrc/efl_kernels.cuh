// efl_kernels.cuh — sm_100a kernels of the per-step Eulerian fluid path.
//
// Each kernel computes what one WGSL entry point of the reference computes
// (file:line cited per kernel), over the same invocation domain, with the
// same floating-point operation order.  The library is built with
// -fmad=false and IEEE division/sqrt so that results are bit-identical to
// the CPU restatement wherever the reference's math is not
// implementation-defined (exp is the only such function on this path).
//
// Device layout: every field is one pitched f32 plane (pitch P floats,
// P = round_up(nx + 1, 32), 128-byte aligned rows).  Cell (x, y), x-face
// (x, y) and y-face (x, y) all live at y * P + x.  Area fractions are kept
// as two face planes fu ((nx+1) x ny) and fv (nx x (ny+1)) instead of the
// reference's per-cell RGBA: the reference computes the fraction of a face
// shared by two cells from the same four level-set samples in the same
// order on both sides, so one value per face is exact and halves the bytes
// the projection reads.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/efl.h"

namespace efl {

#define EFL_DEV __device__ __forceinline__

// Number of kernels this library has launched (all simulations, all
// devices).  Evaluated in every launch configuration as the dynamic
// shared-memory size argument, which it leaves at 0.
uint64_t launches_total();
size_t count_launch();

constexpr float LARGE_FLOAT = 1.0e6f;      // update_solid.wgsl:4, update_fluid_source.wgsl:22
constexpr float FIM_LARGE = 1e30f;         // fast_iterative_method/initialize.wgsl:5
constexpr float FIM_EPS = 1e-6f;           // fast_iterative_method/update.wgsl:9
constexpr float SQRT2_F = 1.41421356237309504880f;
constexpr uint32_t LABEL_NONE = 0, LABEL_SOURCE = 1, LABEL_ACTIVE = 2, LABEL_CONVERGED = 3;

struct Uniform {  // fluid_uniform.wgsl:3-10
    float dx, dt, rho;
    float g[2];
    float m[16];
    float size[2];
};

// A pitched plane with its logical extent.
template <class T>
struct Plane {
    T* p;
    int w, h, P;
    EFL_DEV bool in(int x, int y) const { return (unsigned)x < (unsigned)w && (unsigned)y < (unsigned)h; }
    EFL_DEV T ld(int x, int y) const { return in(x, y) ? p[(size_t)y * P + x] : T{}; }
    EFL_DEV void st(int x, int y, T v) const { if (in(x, y)) p[(size_t)y * P + x] = v; }
    EFL_DEV T& at(int x, int y) const { return p[(size_t)y * P + x]; }
};
using PF = Plane<float>;
using PI = Plane<int32_t>;
using PU = Plane<uint32_t>;
using P2 = Plane<float2>;

// WGSL helpers ---------------------------------------------------------------
EFL_DEV float fclamp01(float v) { return fminf(fmaxf(v, 0.0f), 1.0f); }
EFL_DEV float fclampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
EFL_DEV float wsign(float v) { return v > 0.0f ? 1.0f : (v < 0.0f ? -1.0f : 0.0f); }
EFL_DEV float wlength(float x, float y) { return sqrtf(x * x + y * y); }
// a / b with a selected by the caller: a zero a takes the division's slow path, for the whole warp, so lanes whose
// quotient is not used get another numerator, and the compiler must not see through that selection (20 fixed-count
// iterations at 256^2: 45 -> 33 us).
EFL_DEV float div_any(float a, float b) {
    asm volatile("" : "+f"(a));
    return a / b;
}
// The same for numerators that may be zero themselves: the quotient of a zero is that zero with the product's sign
// (NaN from a NaN or zero b).
EFL_DEV float div_zero(float a, float b) {
    const float q = div_any(a == 0.0f ? 1.0f : a, b);
    const float z = __uint_as_float((__float_as_uint(a) ^ __float_as_uint(b)) & 0x80000000u);
    return a != 0.0f || b != b ? q : b != 0.0f ? z : __int_as_float(0x7fc00000);
}
EFL_DEV float wmix(float a, float b, float t) { return a * (1.0f - t) + b * t; }
EFL_DEV int f2i(float v) { return __float2int_rz(v); }  // truncate, saturate, NaN -> 0
EFL_DEV float2 mat_xy(const float* m, float x, float y) {
    float2 r;
    r.x = ((m[0] * x + m[4] * y) + m[8] * 0.0f) + m[12] * 1.0f;
    r.y = ((m[1] * x + m[5] * y) + m[9] * 0.0f) + m[13] * 1.0f;
    return r;
}
EFL_DEV float det4(const float* m) {
#define A_(r, c) m[(c)*4 + (r)]
    float s0 = A_(0, 0) * A_(1, 1) - A_(1, 0) * A_(0, 1);
    float s1 = A_(0, 0) * A_(1, 2) - A_(1, 0) * A_(0, 2);
    float s2 = A_(0, 0) * A_(1, 3) - A_(1, 0) * A_(0, 3);
    float s3 = A_(0, 1) * A_(1, 2) - A_(1, 1) * A_(0, 2);
    float s4 = A_(0, 1) * A_(1, 3) - A_(1, 1) * A_(0, 3);
    float s5 = A_(0, 2) * A_(1, 3) - A_(1, 2) * A_(0, 3);
    float c5 = A_(2, 2) * A_(3, 3) - A_(3, 2) * A_(2, 3);
    float c4 = A_(2, 1) * A_(3, 3) - A_(3, 1) * A_(2, 3);
    float c3 = A_(2, 1) * A_(3, 2) - A_(3, 1) * A_(2, 2);
    float c2 = A_(2, 0) * A_(3, 3) - A_(3, 0) * A_(2, 3);
    float c1 = A_(2, 0) * A_(3, 2) - A_(3, 0) * A_(2, 2);
    float c0 = A_(2, 0) * A_(3, 1) - A_(3, 0) * A_(2, 1);
#undef A_
    return s0 * c5 - s1 * c4 + s2 * c3 + s3 * c2 - s4 * c1 + s5 * c0;
}

// utils/area_fraction.wgsl:10-12
EFL_DEV float area_fraction(float l0, float l1) { return fclamp01(fmaxf(l0, l1) / fabsf(l0 - l1)); }
// area_fraction(l0, l1) > 0.  The division decides only where its quotient may round to 0 or an operand is not
// finite; otherwise the sign of the larger value does.
EFL_DEV bool area_fraction_positive(float l0, float l1) {
    const float m = fmaxf(l0, l1);
    if (!(m > 0.0f)) return false;  // a NaN operand leaves the other one or NaN: the fraction is 0 or below
    if (m >= 1e-30f && fabsf(l0 - l1) <= 1e8f) return true;
    return area_fraction(l0, l1) > 0.0f;
}
// utils/area_fraction.wgsl:14-56 -> (i-1/2, i+1/2, j-1/2, j+1/2)
EFL_DEV float4 area_fractions(const PF& ls, int x, int y) {
    float c0 = ls.ld(x - 1, y - 1), c1 = ls.ld(x, y - 1), c2 = ls.ld(x + 1, y - 1);
    float c3 = ls.ld(x - 1, y), c4 = ls.ld(x, y), c5 = ls.ld(x + 1, y);
    float c6 = ls.ld(x - 1, y + 1), c7 = ls.ld(x, y + 1), c8 = ls.ld(x + 1, y + 1);
    float mm = 0.25f * (c0 + c1 + c3 + c4);
    float pm = 0.25f * (c1 + c2 + c4 + c5);
    float mp = 0.25f * (c3 + c4 + c6 + c7);
    float pp = 0.25f * (c4 + c5 + c7 + c8);
    return make_float4(area_fraction(mm, mp), area_fraction(pm, pp), area_fraction(mm, pm), area_fraction(mp, pp));
}

// Dispatch-domain helpers (pipeline.rs:175-186).
struct Dom {
    int nx, ny;
    EFL_DEV int cx() const { return (nx / 8) * 8; }
    EFL_DEV int cy() const { return (ny / 8) * 8; }
    EFL_DEV int xrows() const { return (ny / 64) * 64; }
    EFL_DEV int ycols() const { return (nx / 64) * 64; }
};

EFL_DEV int gx() { return blockIdx.x * blockDim.x + threadIdx.x; }
EFL_DEV int gy() { return blockIdx.y * blockDim.y + threadIdx.y; }

// ---------------------------------------------------------------------------
// initialize_grid_center.wgsl:5-15
__global__ void k_init_center(PF ls0, PF ls1, P2 grad, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    float level = (float)(uint32_t)(d.ny - y);
    ls0.st(x, y, level);
    ls1.st(x, y, level);
    grad.st(x, y, make_float2(0.0f, -1.0f));
}
// initialize_grid_edge.wgsl:6-17, (nx+1, ny/64) x (1, 64); v index transposed
__global__ void k_init_edge(PF u0, PF u1, PF v0, PF v1, Dom d) {
    int x = gx(), y = gy();
    if (x > d.nx || y >= d.xrows()) return;
    u0.st(x, y, 0.0f);
    v0.st(y, x, 0.0f);
    u1.st(x, y, 0.0f);
    v1.st(y, x, 0.0f);
}

// update_solid.wgsl:80-85
EFL_DEV float2 to_world(const Uniform& U, float px, float py, int nx, int ny) {
    float uvx = px / (float)nx, uvy = py / (float)ny;
    float xx = (uvx - 0.5f) * U.size[0];
    float yy = (-uvy + 0.5f) * U.size[1];
    return mat_xy(U.m, xx, yy);
}
// update_solid.wgsl:164-175
EFL_DEV float dist_segment(float2 x, float2 a, float2 b) {
    float abx = b.x - a.x, aby = b.y - a.y;
    float t = fclampf(((x.x - a.x) * abx + (x.y - a.y) * aby) / (abx * abx + aby * aby), 0.0f, 1.0f);
    float px = a.x + t * abx, py = a.y + t * aby;
    return wlength(x.x - px, x.y - py);
}
EFL_DEV float dist_sign(float2 x, float2 a, float2 b) {
    float x1x = x.x - a.x, x1y = x.y - a.y;
    float abx = b.x - a.x, aby = b.y - a.y;
    return wsign(x1y * abx - x1x * aby);
}
// update_solid.wgsl:87-109
EFL_DEV float level_rectangle(const efl_solid_obstacle& o, float2 x) {
    float level = LARGE_FLOAT;
    if (det4(o.transform) == 0.0f) return level;
    float2 x0 = mat_xy(o.inverse_transform, x.x, x.y);
    float hx = o.values[0], hy = o.values[1];
    bool ix = fabsf(x0.x) < hx, iy = fabsf(x0.y) < hy;
    if (ix) level = iy ? fmaxf(fabsf(x0.x) - hx, fabsf(x0.y) - hy) : fabsf(x0.y) - hy;
    else level = iy ? fabsf(x0.x) - hx : wlength(fabsf(x0.x) - hx, fabsf(x0.y) - hy);
    return level;
}
// update_solid.wgsl:121-162
EFL_DEV float level_obstacle(const efl_solid_obstacle& o, float2 x) {
    switch (o.shape) {
        case EFL_SHAPE_CIRCLE:
            return wlength(x.x - o.transform[12], x.y - o.transform[13]) - o.values[0];
        case EFL_SHAPE_RECTANGLE:
            return level_rectangle(o, x);
        case EFL_SHAPE_CAPSULE: {
            float2 a = mat_xy(o.transform, o.values[0], o.values[1]);
            float2 b = mat_xy(o.transform, o.values[2], o.values[3]);
            return dist_segment(x, a, b) - o.values[4];
        }
        case EFL_SHAPE_TRIANGLE: {
            float2 p0 = mat_xy(o.transform, o.values[0], o.values[1]);
            float2 p1 = mat_xy(o.transform, o.values[2], o.values[3]);
            float2 p2 = mat_xy(o.transform, o.values[4], o.values[5]);
            float d0 = dist_segment(x, p0, p1), d1 = dist_segment(x, p1, p2), d2 = dist_segment(x, p2, p0);
            float s0 = dist_sign(x, p0, p1), s1 = dist_sign(x, p1, p2), s2 = dist_sign(x, p2, p0);
            float m = fminf(fminf(d0, d1), d2);
            return (s0 > 0.0f && s1 > 0.0f && s2 > 0.0f) ? -m : m;
        }
        default:
            return LARGE_FLOAT;
    }
}
EFL_DEV float2 velocity_at(const efl_solid_obstacle& o, float2 x) {  // update_solid.wgsl:111-119
    float rx = x.x - o.transform[12], ry = x.y - o.transform[13];
    float w = o.angular_velocity;
    return make_float2(o.linear_velocity[0] + -w * ry, o.linear_velocity[1] + w * rx);
}

// update_solid.wgsl:15-78.  Obstacles are staged through shared memory in
// chunks; every invocation walks them in index order as the reference does.
constexpr int OBS_CHUNK = 32;
__global__ void k_update_solid(PF us, PF vs, PF ls_s, PI sid, const efl_solid_obstacle* __restrict__ obs, int n_obs,
                               Uniform U, Dom d) {
    __shared__ efl_solid_obstacle so[OBS_CHUNK];
    int x = gx(), y = gy();
    const int nx = d.nx, ny = d.ny;
    bool active = x < d.cx() && y < d.cy();
    bool border = x == 0 || y == 0 || x == nx - 1 || y == ny - 1;
    float2 xc = to_world(U, (float)x, (float)y, nx, ny);
    float2 xex = to_world(U, (float)x - 0.5f, (float)y - 0.0f, nx, ny);
    float2 xey = to_world(U, (float)x - 0.0f, (float)y - 0.5f, nx, ny);
    int tx = min(x, abs(nx - 1 - x)), ty = min(y, abs(ny - 1 - y));
    float level = (float)min(tx, ty);
    float u = 0.0f, v = 0.0f;
    int32_t id = -1;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int nthreads = blockDim.x * blockDim.y;
    for (int base = 0; base < n_obs; base += OBS_CHUNK) {
        int cnt = min(OBS_CHUNK, n_obs - base);
        __syncthreads();
        const int words = cnt * (int)(sizeof(efl_solid_obstacle) / 4);
        const uint32_t* src = reinterpret_cast<const uint32_t*>(obs + base);
        uint32_t* dst = reinterpret_cast<uint32_t*>(so);
        for (int i = tid; i < words; i += nthreads) dst[i] = src[i];
        __syncthreads();
        if (active && !border) {
            for (int k = 0; k < cnt; ++k) {
                const efl_solid_obstacle& o = so[k];
                float lo = level_obstacle(o, xc);
                if (lo < level) level = lo;
                if (lo < 0.5f) id = (int32_t)o.entity_id;
                float lex = level_obstacle(o, xex);
                if (lex < 0.5f) u = velocity_at(o, xex).x;
                float ley = level_obstacle(o, xey);
                if (ley < 0.5f) v = -velocity_at(o, xey).y;
            }
        }
    }
    if (!active) return;
    if (border) {
        ls_s.st(x, y, 0.0f);
        us.st(x, y, 0.0f);
        vs.st(x, y, 0.0f);
        sid.st(x, y, -1);
        return;
    }
    us.st(x, y, u);
    vs.st(x, y, v);
    ls_s.st(x, y, level);
    sid.st(x, y, id);
}

// update_area_fraction.wgsl:6-14, written as face planes.
__global__ void k_area_fraction(PF ls_s, PF fu, PF fv, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    float4 f = area_fractions(ls_s, x, y);
    fu.st(x, y, f.x);
    fv.st(x, y, f.z);
    if (x == d.nx - 1) fu.st(x + 1, y, f.y);
    if (y == d.ny - 1) fv.st(x, y + 1, f.w);
}

// (i, j), (i + 1, j), (i, j + 1), (i + 1, j + 1), 0 outside: one test for the interior instead of four.
EFL_DEV void load_2x2(const PF& a, int i, int j, float (&q)[4]) {
    if (i >= 0 && j >= 0 && i < a.w - 1 && j < a.h - 1) {
        const float* c = a.p + (size_t)j * a.P + i;
        q[0] = c[0];
        q[1] = c[1];
        q[2] = c[a.P];
        q[3] = c[a.P + 1];
    } else {
        q[0] = a.ld(i, j);
        q[1] = a.ld(i + 1, j);
        q[2] = a.ld(i, j + 1);
        q[3] = a.ld(i + 1, j + 1);
    }
}
// utils/coordinate.wgsl:51-94
EFL_DEV float interp_edge_x(const PF& u, float px, float py) {
    int i = f2i(rintf(px));
    int j = f2i(floorf(py));
    float fi = px + 0.5f - (float)i;
    float fj = py - (float)j;
    float q[4];
    load_2x2(u, i, j, q);
    return wmix(wmix(q[0], q[1], fi), wmix(q[2], q[3], fi), fj);
}
EFL_DEV float interp_edge_y(const PF& v, float px, float py) {
    int i = f2i(floorf(px));
    int j = f2i(rintf(py));
    float fi = px - (float)i;
    float fj = py + 0.5f - (float)j;
    float q[4];
    load_2x2(v, i, j, q);
    return wmix(wmix(q[0], q[1], fi), wmix(q[2], q[3], fi), fj);
}
EFL_DEV float2 runge_kutta(const PF& u, const PF& v, float px, float py, float dt) {
    float vx = interp_edge_x(u, px, py), vy = interp_edge_y(v, px, py);
    float h = 0.5f * dt;
    float mx = px - h * vx, my = py - h * vy;
    float wx = interp_edge_x(u, mx, my), wy = interp_edge_y(v, mx, my);
    return make_float2(px - dt * wx, py - dt * wy);
}
// advect_velocity.wgsl:11-27 (x-major) and :29-45 (y-major)
EFL_DEV float advected_u(const PF& u0, const PF& v0, float dt, int x, int y) {
    float px = (float)x + -0.5f, py = (float)y + 0.0f;
    float2 b = runge_kutta(u0, v0, px, py, dt);
    float dimx = (float)u0.w, dimy = (float)u0.h;
    bool inside = b.x >= 0.0f && b.y >= 0.0f && b.x <= dimx - 1.0f && b.y <= dimy - 1.0f;
    return inside ? interp_edge_x(u0, b.x, b.y) : u0.ld(x, y);
}
EFL_DEV float advected_v(const PF& u0, const PF& v0, float dt, int x, int y) {
    float px = (float)x + 0.0f, py = (float)y + -0.5f;
    float2 b = runge_kutta(u0, v0, px, py, dt);
    float dimx = (float)v0.w, dimy = (float)v0.h;
    bool inside = b.x >= 0.0f && b.y >= 0.0f && b.x <= dimx - 1.0f && b.y <= dimy - 1.0f;
    return inside ? interp_edge_y(v0, b.x, b.y) : v0.ld(x, y);
}
// The faces of each component's dispatch (pipeline.rs:175-186).
template <int COMP>
EFL_DEV bool face_covered(const Dom& d, int x, int y) {
    return COMP == 0 ? x <= d.nx && y < d.xrows() : x < d.ycols() && y <= d.ny;
}
// Both passes in one launch over the larger of their grids: blockIdx.z 0 the x-major faces, 1 the y-major ones.
__global__ void k_advect_uv(PF u0, PF v0, PF u1, PF v1, float dt, Dom d) {
    const int x = gx(), y = gy();
    if (blockIdx.z == 0) {
        if (face_covered<0>(d, x, y)) u1.st(x, y, advected_u(u0, v0, dt, x, y));
    } else {
        if (face_covered<1>(d, x, y)) v1.st(x, y, advected_v(u0, v0, dt, x, y));
    }
}

// exp for the Gaussian force splat.  WGSL's exp is implementation-defined
// (any few-ulp result is conforming), so the library and the CPU oracle both
// evaluate this restatement of the Cody-Waite method: x = k ln2 + r with ln2
// split into an exactly-multipliable high part and a low part, |r| <= ln2/2,
// exp(r) by its degree-7 Taylor polynomial in Horner form (truncation error
// < 1e-8 relative), exact scaling by 2^k.  Within 2 ulp of exp.
EFL_DEV float efl_exp(float x) {
    if (x < -104.0f) return 0.0f;
    if (x > 88.5f) return __int_as_float(0x7f800000);
    float kf = rintf(x * 1.44269504088896341f);
    float r = (x - kf * 0.693145751953125f) - kf * 1.42860682030941723e-6f;
    float p = 1.98412698412698413e-4f;  // 1/7!
    p = p * r + 1.38888888888888889e-3f;
    p = p * r + 8.33333333333333333e-3f;
    p = p * r + 4.16666666666666667e-2f;
    p = p * r + 1.66666666666666667e-1f;
    p = p * r + 0.5f;
    p = p * r + 1.0f;
    p = p * r + 1.0f;
    return ldexpf(p, (int)kf);
}
// apply_forces.wgsl:73-76
EFL_DEV float gaussian_2d(float x, float y, float x0, float y0, float sigma) {
    float b = -1.0f / (2.0f * sigma * sigma);
    float dx = x - x0, dy = y - y0;
    return efl_exp(b * (dx * dx + dy * dy));
}
// area_fraction(l0, l1) == 1, without the division: with m = max(l0, l1) and a = |l0 - l1|, m < a leaves m / a at most
// 1 - 2^-24 (a float below 1), and m >= a > 0 rounds to 1 or above; 0 / 0, inf / inf and NaN give the fraction 0.
EFL_DEV bool area_fraction_one(float l0, float l1) {
    const float m = fmaxf(l0, l1);
    return m >= fabsf(l0 - l1) && m > 0.0f && m < INFINITY;
}
// apply_forces.wgsl:17-43 / 45-71 (comp 0 = u, x-major; comp 1 = v, y-major): whether a face's velocity becomes 0 (all
// air, or solid) ...
template <int COMP>
EFL_DEV bool face_still(const PF& ls0, const PF& face_frac, int x, int y, const Dom& d) {
    // af(idx).x / af(idx).z; outside the cell texture the reference reads 0,
    // and the face planes hold 0 there too (border faces of the solid ring).
    if (!(x < d.nx && y < d.ny) || face_frac.at(x, y) == 0.0f) return true;
    // The corners of the face (area_fractions): u faces use the columns x - 1 and x, v faces the rows y - 1 and y.
    float m0, m1;
    if (COMP == 0) {
        const float c0 = ls0.ld(x - 1, y - 1), c1 = ls0.ld(x, y - 1), c3 = ls0.ld(x - 1, y), c4 = ls0.at(x, y);
        const float c6 = ls0.ld(x - 1, y + 1), c7 = ls0.ld(x, y + 1);
        m0 = 0.25f * (c0 + c1 + c3 + c4);
        m1 = 0.25f * (c3 + c4 + c6 + c7);
    } else {
        const float c0 = ls0.ld(x - 1, y - 1), c1 = ls0.ld(x, y - 1), c2 = ls0.ld(x + 1, y - 1);
        const float c3 = ls0.ld(x - 1, y), c4 = ls0.at(x, y), c5 = ls0.ld(x + 1, y);
        m0 = 0.25f * (c0 + c1 + c3 + c4);
        m1 = 0.25f * (c1 + c2 + c4 + c5);
    }
    return area_fraction_one(m0, m1);
}
// ... and the velocity of the others.
template <int COMP>
EFL_DEV float forced(float val, const efl_force* __restrict__ forces, int n_forces, const Uniform& U, int x, int y) {
    float net = U.g[COMP];
    for (int n = n_forces; n > 0; --n) {
        const efl_force F = forces[n - 1];
        net = net + F.force[COMP] * gaussian_2d((float)x, (float)y, F.position[0], F.position[1], 10.0f);
    }
    return val + net * U.dt / U.dx;
}
template <int COMP>
EFL_DEV void apply_forces_at(const PF& vel, const PF& ls0, const PF& face_frac, const efl_force* __restrict__ forces,
                             int n_forces, const Uniform& U, const Dom& d) {
    const int x = gx(), y = gy();
    if (!face_covered<COMP>(d, x, y)) return;
    vel.st(x, y, face_still<COMP>(ls0, face_frac, x, y, d) ? 0.0f
                                                           : forced<COMP>(vel.ld(x, y), forces, n_forces, U, x, y));
}
// Both components in one launch over the larger of their grids (blockIdx.z: 0 = u, 1 = v).
__global__ void k_apply_forces_uv(PF u, PF v, PF ls0, PF fu, PF fv, const efl_force* __restrict__ forces, int n_forces,
                                  Uniform U, Dom d) {
    if (blockIdx.z == 0)
        apply_forces_at<0>(u, ls0, fu, forces, n_forces, U, d);
    else
        apply_forces_at<1>(v, ls0, fv, forces, n_forces, U, d);
}

// Advection and forces in one pass, as a step runs them one after the other: the advected velocity is neither written
// nor read back, and faces that the forces set to 0 (air and solid: most of a dam break) are not advected at all
// (4096^2: 329 + 247 us before).
__global__ void k_advect_forces_uv(PF u0, PF v0, PF u1, PF v1, PF ls0, PF fu, PF fv,
                                   const efl_force* __restrict__ forces, int n_forces, Uniform U, Dom d) {
    const int x = gx(), y = gy();
    if (blockIdx.z == 0) {
        if (!face_covered<0>(d, x, y)) return;
        u1.st(x, y, face_still<0>(ls0, fu, x, y, d)
                        ? 0.0f
                        : forced<0>(advected_u(u0, v0, U.dt, x, y), forces, n_forces, U, x, y));
    } else {
        if (!face_covered<1>(d, x, y)) return;
        v1.st(x, y, face_still<1>(ls0, fv, x, y, d)
                        ? 0.0f
                        : forced<1>(advected_v(u0, v0, U.dt, x, y), forces, n_forces, U, x, y));
    }
}

// divergence.wgsl:16-42 (fractions of levelset_solid = the face planes)
__global__ void k_divergence(PF u1, PF v1, PF us, PF vs, PF fu, PF fv, PF div, float dx, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    float fx0 = fu.ld(x, y), fx1 = fu.ld(x + 1, y), fy0 = fv.ld(x, y), fy1 = fv.ld(x, y + 1);
    float u_ij = u1.ld(x, y), u_ip = u1.ld(x + 1, y);
    float v_ij = v1.ld(x, y), v_jp = v1.ld(x, y + 1);
    float du_f = fx1 * u_ip - fx0 * u_ij;
    float dv_f = fy1 * v_jp - fy0 * v_ij;
    float us_m = us.ld(x, y), us_p = us.ld(x + 1, y);
    float vs_m = vs.ld(x, y), vs_p = vs.ld(x, y + 1);
    float du_s = (1.0f - fx1) * us_p - (1.0f - fx0) * us_m;
    float dv_s = (1.0f - fy1) * vs_p - (1.0f - fy0) * vs_m;
    div.st(x, y, -(du_f + dv_f + du_s + dv_s) / dx);
}

// Which 32 x 8 blocks of cells hold a cell with level set < 0 (one CTA per block).  The large solves skip the others
// (dam breaks and pools are half air or more): their correction, residual and weights are 0.
__global__ void __launch_bounds__(256) k_wet_blocks(PF ls, unsigned char* wet) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    const int any = __syncthreads_or(x < ls.w && y < ls.h && ls.at(x, y) < 0.0f);
    if (threadIdx.x == 0 && threadIdx.y == 0) wet[blockIdx.y * gridDim.x + blockIdx.x] = any != 0;
}
// The same for the next coarser level, from the finer one's (fw x fh blocks): a coarse cell is water only if one of its
// children is (restriction.wgsl takes a child's level set).
__global__ void k_wet_coarsen(const unsigned char* fine, int fw, int fh, unsigned char* wet, int w, int h) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    unsigned any = 0;
    for (int j = 0; j < 2; ++j)
        for (int i = 0; i < 2; ++i)
            if (2 * x + i < fw && 2 * y + j < fh) any |= fine[(2 * y + j) * fw + 2 * x + i];
    wet[y * w + x] = any != 0;
}
// The tiles of 64 x 32 cells with a wet block, list[0 .. count), and the others, list[count .. ntiles), each in any
// order.  counts[2] = 0 before.
__global__ void k_wet_tiles(const unsigned char* wet, int w, int h, int tiles_x, int ntiles, int* list, int* counts) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    bool any = false;
    if (t < ntiles) {
        const int bx = (t % tiles_x) * 2, by = (t / tiles_x) * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) any |= bx + i < w && by + j < h && wet[(by + j) * w + bx + i];
    }
    const unsigned hot = __ballot_sync(0xffffffffu, any), cold = __ballot_sync(0xffffffffu, t < ntiles && !any);
    int at[2] = {0, 0};
    if (lane == 0) {
        if (hot) at[0] = atomicAdd(&counts[0], __popc(hot));
        if (cold) at[1] = atomicAdd(&counts[1], __popc(cold));
    }
    at[0] = __shfl_sync(0xffffffffu, at[0], 0);
    at[1] = __shfl_sync(0xffffffffu, at[1], 0);
    const unsigned below = (1u << lane) - 1u;
    if (any) list[at[0] + __popc(hot & below)] = t;
    else if (t < ntiles) list[ntiles - 1 - (at[1] + __popc(cold & below))] = t;
}

// One level of the pressure system: iterate x, right-hand side b and
// residual r of type T (f32: the reference's fixed-count solve; f64: the
// tolerance-driven solve), with the level's f32 air level set and face
// fractions.
template <class T>
struct LevelT {
    Plane<T> x, b, r;
    PF ls, fu, fv;
    int nx, ny;
};
using Level = LevelT<float>;
using Level64 = LevelT<double>;

// projection/shaders/gauss_seidel.wgsl:44-88.  T = float is the reference's
// arithmetic; T = double evaluates the same expression tree in f64 from the
// f32 inputs.
template <class T>
EFL_DEV T gs_update(const LevelT<T>& L, T c_div, T weight, int x, int y) {
    float lij = L.ls.at(x, y);
    if (lij >= 0.0f) return T(0);
    float f0 = L.fu.at(x, y), f1 = L.fu.at(x + 1, y), f2 = L.fv.at(x, y), f3 = L.fv.at(x, y + 1);
    T p_old = L.x.at(x, y);
    if (f0 == 0.0f && f1 == 0.0f && f2 == 0.0f && f3 == 0.0f) return T(0);
    T denom = T(0);
    T nume = c_div * L.b.at(x, y);
    const int ox[4] = {-1, 1, 0, 0}, oy[4] = {0, 0, -1, 1};
    const T fvv[4] = {(T)f0, (T)f1, (T)f2, (T)f3};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int jx = x + ox[i], jy = y + oy[i];
        if ((unsigned)jx < (unsigned)L.nx && (unsigned)jy < (unsigned)L.ny) {
            float level = L.ls.at(jx, jy);
            if (level < 0.0f) {
                denom += fvv[i];
                nume += fvv[i] * L.x.at(jx, jy);
            } else {
                denom += fvv[i] * (T(1) - (T)level / (T)lij);
            }
        }
    }
    if (fabs(denom) < (T)1.0e-6f) return T(0);
    // f32: the reference's division; f64 (tolerance-driven, an extension):
    // nume * (1/denom), the form the persistent solver evaluates.
    T p_new;
    if constexpr (sizeof(T) == 8) p_new = nume * (T(1) / denom);
    else p_new = nume / denom;
    return weight * p_new + (T(1) - weight) * p_old;
}
// ((dx*dx)*rho)/dt as gauss_seidel.wgsl:58 evaluates it, dx = resolution_scale*dx.
template <class T>
EFL_DEV T gs_cdiv(float dx_scaled, float rho, float dt) {
    T d = (T)dx_scaled;
    return d * d * (T)rho / (T)dt;
}
// gauss_seidel.wgsl:12-42: colour 1 = red ((x+y) odd), 0 = black.  One
// thread per cell of the colour.  wet (or null): blocks without water are skipped (their iterate is 0 already).
template <class T>
__global__ void k_gs_color(LevelT<T> L, float dx_scaled, float rho, float dt, float weight, int color,
                           const unsigned char* wet = nullptr) {
    int tx = gx(), y = gy();
    if (wet) {  // a CTA's 64 x 8 cells
        const int w = (L.nx + 31) / 32, b = blockIdx.y * w + 2 * blockIdx.x;
        if (!wet[b] && !(2 * (int)blockIdx.x + 1 < w && wet[b + 1])) return;
    }
    int x = 2 * tx + ((y + color) & 1);
    if (x >= L.nx || y >= L.ny) return;
    L.x.at(x, y) = gs_update(L, gs_cdiv<T>(dx_scaled, rho, dt), (T)weight, x, y);
}

// n (1 or 2) red-black iterations of a V-cycle's smoother (weight 1) in one pass from L.x to `out`: gs_update on
// 32 x 32 tiles with a halo of 4 cells, a thread per 2 x 2 block, its coefficients in registers and the image of x in
// shared memory by colour.  Cells of the image's outermost ring update from clamped neighbours: what is wrong moves
// inwards a ring per half-sweep and stays in the halo.  A launch per half-sweep read every plane and divided in every
// cell each time: 149 us of a V-cycle on the levels 2048^2 to 512^2 in f64 (half of them water), 127 here (latency of
// the first loads, two CTAs per SM); 46 and 27 us in f32 on 768 x 512 and 384 x 256.  wet (or null): tiles without water are skipped, zero in both planes already.
constexpr int GT_E = 40, GT_H = 4, GT_O = GT_E - 2 * GT_H, GT_B = GT_E / 2, GT_NT = 416, GT_WP = 26;
template <class T>
__global__ void __launch_bounds__(GT_NT, 2) k_gs_tile(LevelT<T> L, Plane<T> out, float dx_scaled, float rho, float dt,
                                                       int first, int n, const unsigned char* wet) {
    static_assert(GT_B * GT_B <= GT_NT && GT_O == 32, "a thread per block; four 32 x 8 blocks of wet per tile");
    __shared__ T xs[2][GT_E][GT_WP];  // [k][y][x / 2], k = (x + y) & 1 (1: red)
    if (wet) {
        const int w = (L.nx + 31) / 32, h = (L.ny + 7) / 8;
        unsigned any = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int by = 4 * (int)blockIdx.y + j;
            any |= by < h ? wet[by * w + blockIdx.x] : 0u;
        }
        if (!any) return;
    }
    const bool active = threadIdx.x < GT_B * GT_B;
    const int bx = active ? (int)threadIdx.x % GT_B : 0, by = active ? (int)threadIdx.x / GT_B : 0;
    const int gx0 = (int)blockIdx.x * GT_O - GT_H + 2 * bx, gy0 = (int)blockIdx.y * GT_O - GT_H + 2 * by;
    // every load of the block first, at clamped places
    float lv[4][4], fu[2][3], fv[3][2];
    T pv[4], cb[4], inv[4];  // inv: 1 / denom in f64, denom in f32 (gs_update)
    {
        int xc[4], yc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xc[i] = min(max(gx0 - 1 + i, 0), L.nx - 1);
            yc[i] = min(max(gy0 - 1 + i, 0), L.ny - 1);
        }
        const int fx[3] = {xc[1], min(max(gx0 + 1, 0), L.nx), min(max(gx0 + 2, 0), L.nx)};
        const int fy[3] = {yc[1], min(max(gy0 + 1, 0), L.ny), min(max(gy0 + 2, 0), L.ny)};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == 1 || i == 2 || j == 1 || j == 2) lv[j][i] = L.ls.at(xc[i], yc[j]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                pv[2 * j + i] = L.x.at(xc[1 + i], yc[1 + j]);
                cb[2 * j + i] = L.b.at(xc[1 + i], yc[1 + j]);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                fu[j][i] = L.fu.at(fx[i], yc[1 + j]);
                fv[i][j] = L.fv.at(xc[1 + j], fy[i]);
            }
        }
    }
    const T c_div = gs_cdiv<T>(dx_scaled, rho, dt);
    float w[4][4];
    unsigned upd = 0, in = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int qx = q & 1, qy = q >> 1, gx = gx0 + qx, gy = gy0 + qy;
        const float f[4] = {fu[qy][qx], fu[qy][qx + 1], fv[qy][qx], fv[qy + 1][qx]};
        const float ln[4] = {lv[1 + qy][qx], lv[1 + qy][qx + 2], lv[qy][1 + qx], lv[qy + 2][1 + qx]};
        const bool nb[4] = {gx > 0, gx + 1 < L.nx, gy > 0, gy + 1 < L.ny};
        const float lij = lv[1 + qy][1 + qx];
        T denom = T(0);
#pragma unroll
        for (int k = 0; k < 4; ++k) w[q][k] = 0.0f;
        if (active && (unsigned)gx < (unsigned)L.nx && (unsigned)gy < (unsigned)L.ny) {
            in |= 1u << q;
            if (!(lij >= 0.0f) && !(f[0] == 0.0f && f[1] == 0.0f && f[2] == 0.0f && f[3] == 0.0f)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (!nb[k]) continue;
                    if (ln[k] < 0.0f) {
                        denom += (T)f[k];
                        w[q][k] = f[k];
                    } else {
                        denom += (T)f[k] * (T(1) - (T)ln[k] / (T)lij);
                    }
                }
                if (!(fabs(denom) < (T)1.0e-6f)) upd |= 1u << q;
            }
        } else {
            pv[q] = T(0);
        }
        const bool u = (upd >> q) & 1u;
        cb[q] = u ? c_div * cb[q] : T(0);
        inv[q] = u ? denom : T(1);
        if constexpr (sizeof(T) == 8) inv[q] = T(1) / inv[q];
        if (active) xs[(qx + qy) & 1][2 * by + qy][bx] = pv[q];
    }
    __syncthreads();
    const int r0 = 2 * by, r1 = r0 + 1, up = max(r0 - 1, 0), dn = min(r1 + 1, GT_E - 1);
    const int lf = max(bx - 1, 0), rt = min(bx + 1, GT_B - 1);
    auto cell = [&](int q, T l, T r, T u, T d) {
        T nume = cb[q];
        nume = nume + (T)w[q][0] * l;
        nume = nume + (T)w[q][1] * r;
        nume = nume + (T)w[q][2] * u;
        nume = nume + (T)w[q][3] * d;
        const bool up_ = (upd >> q) & 1u;
        T pn;
        if constexpr (sizeof(T) == 8) pn = nume * inv[q];
        else pn = div_zero(up_ ? nume : 1.0f, inv[q]);
        pv[q] = up_ ? T(1) * pn + T(0) * pv[q] : T(0);
    };
    for (int h = 0; h < 2 * n; ++h) {
        if ((first ^ h) & 1) {  // red: cells 1 and 2
            const T r = xs[0][r0][rt], u = xs[0][up][bx], l = xs[0][r1][lf], d = xs[0][dn][bx];
            cell(1, pv[0], r, u, pv[3]);
            cell(2, l, pv[3], pv[0], d);
            if (active) {
                xs[1][r0][bx] = pv[1];
                xs[1][r1][bx] = pv[2];
            }
        } else {  // black: cells 0 and 3
            const T l = xs[1][r0][lf], u = xs[1][up][bx], r = xs[1][r1][rt], d = xs[1][dn][bx];
            cell(0, l, pv[1], u, pv[2]);
            cell(3, pv[2], r, pv[1], d);
            if (active) {
                xs[0][r0][bx] = pv[0];
                xs[0][r1][bx] = pv[3];
            }
        }
        __syncthreads();
    }
    constexpr int B0 = GT_H / 2, B1 = B0 + GT_O / 2;
    if (!active || bx < B0 || bx >= B1 || by < B0 || by >= B1) return;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if ((in >> q) & 1u) out.at(gx0 + (q & 1), gy0 + (q >> 1)) = pv[q];
}

// projection/shaders/residual.wgsl:12-57
template <class T>
EFL_DEV T residual_factor(float dt, float rho, float dx_scaled) {
    T d = (T)dx_scaled;
    return (T)dt / (T)rho / d / d;
}
// f32: the reference's operation order.  f64: the same operator in
// factored form r = b - factor * (denom * x - sum_fluid f * x_nb), denom
// accumulated in the reference's neighbour order.
template <class T>
EFL_DEV T residual_at(const LevelT<T>& L, T factor, int x, int y, bool* counted) {
    *counted = false;
    float phi = L.ls.at(x, y);
    if (phi >= 0.0f) return T(0);
    float f0 = L.fu.at(x, y), f1 = L.fu.at(x + 1, y), f2 = L.fv.at(x, y), f3 = L.fv.at(x, y + 1);
    if (f0 == 0.0f && f1 == 0.0f && f2 == 0.0f && f3 == 0.0f) return T(0);
    *counted = true;
    T xc = L.x.at(x, y);
    const int ox[4] = {-1, 1, 0, 0}, oy[4] = {0, 0, -1, 1};
    const T fvv[4] = {(T)f0, (T)f1, (T)f2, (T)f3};
    if constexpr (sizeof(T) == 8) {
        T denom = T(0), sum = T(0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int jx = x + ox[i], jy = y + oy[i];
            if ((unsigned)jx < (unsigned)L.nx && (unsigned)jy < (unsigned)L.ny) {
                float pn = L.ls.at(jx, jy);
                if (pn < 0.0f) {
                    denom += fvv[i];
                    sum += fvv[i] * L.x.at(jx, jy);
                } else {
                    denom += fvv[i] * (T(1) - (T)pn / (T)phi);
                }
            }
        }
        return L.b.at(x, y) - factor * (denom * xc - sum);
    } else {
        T r = L.b.at(x, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int jx = x + ox[i], jy = y + oy[i];
            if ((unsigned)jx < (unsigned)L.nx && (unsigned)jy < (unsigned)L.ny) {
                float pn = L.ls.at(jx, jy);
                if (pn < 0.0f) r -= fvv[i] * (xc - L.x.at(jx, jy)) * factor;
                else r -= fvv[i] * (T(1) - (T)pn / (T)phi) * xc * factor;
            }
        }
        return r;
    }
}
template <class T>
__global__ void k_residual(LevelT<T> L, float dt, float rho, float dx_scaled) {
    int x = gx(), y = gy();
    if (x >= L.nx || y >= L.ny) return;
    bool c;
    L.r.at(x, y) = residual_at(L, residual_factor<T>(dt, rho, dx_scaled), x, y, &c);
}
// restriction.wgsl:10-60 (the fractions on face planes)
// The coarse cell (x, y) from its four children's residuals r(2x + i, 2y + j) = rij (0 outside the level).
template <class T>
EFL_DEV void restrict_from(const LevelT<T>& F, const LevelT<T>& C, int x, int y, T r00, T r01, T r10, T r11) {
    int fx = 2 * x, fy = 2 * y;
    T br = T(0.25) * (r00 + r01 + r10 + r11);
    float ph0 = F.ls.ld(fx, fy), ph1 = F.ls.ld(fx, fy + 1), ph2 = F.ls.ld(fx + 1, fy), ph3 = F.ls.ld(fx + 1, fy + 1);
    float pr = ph0;
    if (fabsf(ph1) < fabsf(pr)) pr = ph1;
    if (fabsf(ph2) < fabsf(pr)) pr = ph2;
    if (fabsf(ph3) < fabsf(pr)) pr = ph3;
    C.b.at(x, y) = br;
    C.ls.at(x, y) = pr;
    C.fu.at(x, y) = 0.5f * (F.fu.ld(fx, fy) + F.fu.ld(fx, fy + 1));
    C.fv.at(x, y) = 0.5f * (F.fv.ld(fx, fy) + F.fv.ld(fx + 1, fy));
    if (x == C.nx - 1) C.fu.at(x + 1, y) = 0.5f * (F.fu.ld(fx + 2, fy) + F.fu.ld(fx + 2, fy + 1));
    if (y == C.ny - 1) C.fv.at(x, y + 1) = 0.5f * (F.fv.ld(fx, fy + 2) + F.fv.ld(fx + 1, fy + 2));
    C.x.at(x, y) = T(0);
}
template <class T>
EFL_DEV void restrict_cell(const LevelT<T>& F, const LevelT<T>& C, int x, int y) {
    int fx = 2 * x, fy = 2 * y;
    restrict_from(F, C, x, y, F.r.ld(fx, fy), F.r.ld(fx, fy + 1), F.r.ld(fx + 1, fy), F.r.ld(fx + 1, fy + 1));
}
// The residual (k_residual) and the restriction in one pass: each coarse cell computes its four children's
// residuals (residual_at, 0 outside the level, as the residual plane reads there) and restricts them, so the
// fine residual plane is neither written nor read back.  The same values, in the same order.  wet: C's wet blocks in a
// solve's later V-cycles (null in the first one), when C's geometry is known and blocks without water hold zeros.
template <class T>
__global__ void k_residual_restrict(LevelT<T> F, LevelT<T> C, float dt, float rho, float dx_scaled,
                                    const unsigned char* wet = nullptr) {
    int x = gx(), y = gy();
    if (wet && !wet[blockIdx.y * gridDim.x + blockIdx.x]) return;
    if (x >= C.nx || y >= C.ny) return;
    const T fac = residual_factor<T>(dt, rho, dx_scaled);
    auto rr = [&](int ax, int ay) -> T {
        bool c;
        return (ax < F.nx && ay < F.ny) ? residual_at(F, fac, ax, ay, &c) : T(0);
    };
    const int fx = 2 * x, fy = 2 * y;
    const T r00 = rr(fx, fy), r01 = rr(fx, fy + 1), r10 = rr(fx + 1, fy), r11 = rr(fx + 1, fy + 1);
    if (wet) {
        C.b.at(x, y) = T(0.25) * (r00 + r01 + r10 + r11);
        C.x.at(x, y) = T(0);
        return;
    }
    restrict_from(F, C, x, y, r00, r01, r10, r11);
}
// prolongation.wgsl:5-34
template <class T>
EFL_DEV void prolong_cell(const LevelT<T>& F, const LevelT<T>& C, int x, int y) {
    T corr = C.x.at(x, y);
    const int ox[4] = {0, 1, 0, 1}, oy[4] = {0, 0, 1, 1};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int fx = 2 * x + ox[i], fy = 2 * y + oy[i];
        if (F.ls.ld(fx, fy) < 0.0f && F.x.in(fx, fy)) F.x.at(fx, fy) = corr + F.x.at(fx, fy);
    }
}
template <class T>
__global__ void k_prolongation(LevelT<T> F, LevelT<T> C, const unsigned char* wet = nullptr) {  // wet: C's blocks
    int x = gx(), y = gy();
    if (wet && !wet[blockIdx.y * gridDim.x + blockIdx.x]) return;
    if (x >= C.nx || y >= C.ny) return;
    prolong_cell(F, C, x, y);
}

// The coarse tail of a V-cycle (multi_grid.rs:390-475) in ONE launch of one
// CTA: every level from `first` down (each at most VT_MAX_CELLS cells, held
// in L2) with block barriers between the steps instead of a launch per
// half-sweep, residual, restriction and prolongation.  Same per-cell
// functions and the same step order as the launch-per-step form (smoother
// weight 1, resolution scale 2^level; `symmetric`: post-smoothing black then
// red), so the result is identical.
constexpr int VT_THREADS = 1024, VT_MAX_LEVELS = 14;
constexpr int VT_MAX_CELLS = 128 * 128;
template <class T>
struct VTailArgs {
    LevelT<T> lv[VT_MAX_LEVELS];
    int first, count;  // levels first .. count - 1
    float dx, rho, dt;
    int pre, post, coarsest, symmetric;
};
template <class T>
EFL_DEV void vt_sweeps(const LevelT<T>& L, float dxs, float rho, float dt, int n, int c0) {
    const T cd = gs_cdiv<T>(dxs, rho, dt);
    const int hw = (L.nx + 1) / 2;
    for (int k = 0; k < n; ++k) {
        for (int h = 0; h < 2; ++h) {
            const int color = h == 0 ? c0 : 1 - c0;
            for (int i = threadIdx.x; i < hw * L.ny; i += VT_THREADS) {
                const int y = i / hw, x = 2 * (i - y * hw) + ((y + color) & 1);
                if (x < L.nx) L.x.at(x, y) = gs_update(L, cd, T(1), x, y);
            }
            __syncthreads();
        }
    }
}
template <class T>
__global__ void __launch_bounds__(VT_THREADS, 1) k_vcycle_tail(VTailArgs<T> a) {
    const int last = a.count - 1;
    // down: pre-smoothing, residual, restriction
    for (int i = a.first; i < last; ++i) {
        const LevelT<T>& L = a.lv[i];
        const LevelT<T>& C = a.lv[i + 1];
        const float dxs = (float)(1u << i) * a.dx;
        vt_sweeps(L, dxs, a.rho, a.dt, a.pre, 1);
        const T fac = residual_factor<T>(a.dt, a.rho, dxs);
        for (int j = threadIdx.x; j < L.nx * L.ny; j += VT_THREADS) {
            const int y = j / L.nx, x = j - y * L.nx;
            bool c;
            L.r.at(x, y) = residual_at(L, fac, x, y, &c);
        }
        __syncthreads();
        for (int j = threadIdx.x; j < C.nx * C.ny; j += VT_THREADS) {
            const int y = j / C.nx;
            restrict_cell(L, C, j - y * C.nx, y);
        }
        __syncthreads();
    }
    vt_sweeps(a.lv[last], (float)(1u << last) * a.dx, a.rho, a.dt, a.coarsest, 1);
    // up: prolongation, post-smoothing
    for (int i = last - 1; i >= a.first; --i) {
        const LevelT<T>& L = a.lv[i];
        const LevelT<T>& C = a.lv[i + 1];
        for (int j = threadIdx.x; j < C.nx * C.ny; j += VT_THREADS) {
            const int y = j / C.nx;
            prolong_cell(L, C, j - y * C.nx, y);
        }
        __syncthreads();
        vt_sweeps(L, (float)(1u << i) * a.dx, a.rho, a.dt, a.post, a.symmetric ? 0 : 1);
    }
}

// Residual norms ||r||^2, ||b||^2 over cells with phi < 0 that are not
// fully solid; FP64, warp-shuffle + block reduction, per-block partials
// summed in block order by k_norm_finalize (deterministic).
constexpr int NORM_THREADS = 256;
EFL_DEV double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// Latency of dependent loads bounds it, so all of its (at most 1024) blocks are resident at once, 7 per SM: 45 -> 31 us
// at 2048^2 in f64, where 57 registers had allowed 4.
template <class T>
__global__ void __launch_bounds__(NORM_THREADS, 7)
    k_residual_norm(LevelT<T> L, float dt, float rho, float dx, double2* partials) {
    __shared__ double sr[NORM_THREADS / 32], sb[NORM_THREADS / 32];
    const T factor = residual_factor<T>(dt, rho, dx);
    const int n = L.nx * L.ny;
    double ar = 0.0, ab = 0.0;
    for (int i = blockIdx.x * NORM_THREADS + threadIdx.x; i < n; i += gridDim.x * NORM_THREADS) {
        int y = i / L.nx, x = i - y * L.nx;
        bool c;
        T r = residual_at(L, factor, x, y, &c);
        if (c) {
            double b = (double)L.b.at(x, y);
            ar += (double)r * (double)r;
            ab += b * b;
        }
    }
    ar = warp_sum(ar);
    ab = warp_sum(ab);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        sr[w] = ar;
        sb[w] = ab;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tr = 0.0, tb = 0.0;
        for (int k = 0; k < NORM_THREADS / 32; ++k) {
            tr += sr[k];
            tb += sb[k];
        }
        partials[blockIdx.x] = make_double2(tr, tb);
    }
}
// Post-projection divergence diagnostic: the operator of divergence.wgsl:16-42
// applied to the projected velocity (u0, v0) at the cells the residual
// counts (phi < 0, not fully solid).  Per block: x = FP64 sum of squares,
// y = the largest magnitude; k_div_norm_finalize sums x in block order and
// takes the maximum of y (deterministic).
__global__ void __launch_bounds__(NORM_THREADS)
    k_divergence_norm(PF u0, PF v0, PF us, PF vs, PF fu, PF fv, PF ls0, float dx, Dom d, double2* partials) {
    __shared__ double ss[NORM_THREADS / 32], sm[NORM_THREADS / 32];
    const int n = d.nx * d.ny;
    double a2 = 0.0, amax = 0.0;
    for (int i = blockIdx.x * NORM_THREADS + threadIdx.x; i < n; i += gridDim.x * NORM_THREADS) {
        const int y = i / d.nx, x = i - y * d.nx;
        if (!(ls0.at(x, y) < 0.0f)) continue;
        const float fx0 = fu.ld(x, y), fx1 = fu.ld(x + 1, y), fy0 = fv.ld(x, y), fy1 = fv.ld(x, y + 1);
        if (fx0 == 0.0f && fx1 == 0.0f && fy0 == 0.0f && fy1 == 0.0f) continue;
        const float du_f = fx1 * u0.ld(x + 1, y) - fx0 * u0.ld(x, y);
        const float dv_f = fy1 * v0.ld(x, y + 1) - fy0 * v0.ld(x, y);
        const float du_s = (1.0f - fx1) * us.ld(x + 1, y) - (1.0f - fx0) * us.ld(x, y);
        const float dv_s = (1.0f - fy1) * vs.ld(x, y + 1) - (1.0f - fy0) * vs.ld(x, y);
        const double dv = (double)(-(du_f + dv_f + du_s + dv_s) / dx);
        a2 += dv * dv;
        amax = fmax(amax, fabs(dv));
    }
    a2 = warp_sum(a2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_down_sync(0xffffffffu, amax, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        ss[w] = a2;
        sm[w] = amax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t2 = 0.0, tm = 0.0;
        for (int k = 0; k < NORM_THREADS / 32; ++k) {
            t2 += ss[k];
            tm = fmax(tm, sm[k]);
        }
        partials[blockIdx.x] = make_double2(t2, tm);
    }
}
__global__ void k_div_norm_finalize(const double2* partials, int n, double* out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double a2 = 0.0, m = 0.0;
    for (int i = 0; i < n; ++i) {
        a2 += partials[i].x;
        m = fmax(m, partials[i].y);
    }
    out[0] = a2;
    out[1] = m;
}
// The partials in block order, r and b by a thread each (one CTA of NORM_THREADS; n <= 1024).  The sums are one chain of
// dependent additions; the loads are not (one thread for all took 50 us at 1024 partials, 76 times a solve).
__global__ void __launch_bounds__(NORM_THREADS) k_norm_finalize(const double2* partials, int n, double* out) {
    __shared__ double sp[2][1024];
    for (int i = threadIdx.x; i < n; i += NORM_THREADS) {
        const double2 v = partials[i];
        sp[0][i] = v.x;
        sp[1][i] = v.y;
    }
    __syncthreads();
    if (threadIdx.x == 0 || threadIdx.x == 32) {
        const double* p = sp[threadIdx.x >> 5];
        double a = 0.0;
#pragma unroll 8
        for (int i = 0; i < n; ++i) a += p[i];
        out[threadIdx.x >> 5] = a;
    }
}
// f32 <-> f64 transfers of the tolerance-driven solve.
__global__ void k_widen(PF p0, PF div, Plane<double> x, Plane<double> b) {
    int i = gx(), y = gy();
    if (i >= p0.w || y >= p0.h) return;
    x.at(i, y) = (double)p0.at(i, y);
    b.at(i, y) = (double)div.at(i, y);
}
__global__ void k_narrow(Plane<double> x, PF p0) {
    int i = gx(), y = gy();
    if (i >= p0.w || y >= p0.h) return;
    p0.at(i, y) = (float)x.at(i, y);
}

// shaders/jacobi_iteration.wgsl:39-91 (levelset_solid fractions = face planes), JC_K iterations per launch: a CTA
// holds its 32 x 32 cells with a halo of JC_K cells in shared memory (an iteration reads radius 1, so after JC_K of
// them the owned cells are exact), each thread the coefficients of its cells in registers.  The reference's 100
// iterations as a launch each were bound by their launches on small grids (2.6 us of kernel and about 1 us of gap at
// 200 x 136: 360 us) and by passes over memory on large ones; ten per launch take 16.5 us, most of it the cells' chains
// of sums and a division, and read the grid once.
constexpr int JC_T = 32, JC_K = 10, JC_E = JC_T + 2 * JC_K, JC_P = JC_E + 2, JC_THREADS = 1024;
__global__ void __launch_bounds__(JC_THREADS) k_jacobi(PF p_in, PF p_out, PF ls0, PF fu, PF fv, PF div, Uniform U, Dom d) {
    constexpr int N = JC_E * JC_E, PER = (N + JC_THREADS - 1) / JC_THREADS;
    __shared__ float sp[2][JC_P * JC_P];  // with a ring of zeros
    const int x0 = blockIdx.x * JC_T - JC_K, y0 = blockIdx.y * JC_T - JC_K;
    // Every load of the tile in flight at once: the level set with a ring (into the second image first), then the
    // cells' pressure, fractions and divergence; 0 outside the domain.
    float ring[(JC_P * JC_P + JC_THREADS - 1) / JC_THREADS];
#pragma unroll
    for (int k = 0; k < (JC_P * JC_P + JC_THREADS - 1) / JC_THREADS; ++k) {
        const int i = threadIdx.x + k * JC_THREADS;
        ring[k] = i < JC_P * JC_P ? ls0.ld(x0 - 1 + i % JC_P, y0 - 1 + i / JC_P) : 0.0f;
    }
    float w[PER][4], coef[PER], rhs[PER], pv[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = threadIdx.x + k * JC_THREADS, ly = i / JC_E, lx = i - ly * JC_E, x = x0 + lx, y = y0 + ly;
        const bool in = i < N && x >= 0 && y >= 0 && x < d.cx() && y < d.cy();
        pv[k] = in ? p_in.at(x, y) : 0.0f;
        rhs[k] = in ? div.at(x, y) : 0.0f;
        w[k][0] = in ? fu.at(x, y) : 0.0f;
        w[k][1] = in ? fu.at(x + 1, y) : 0.0f;
        w[k][2] = in ? fv.at(x, y) : 0.0f;
        w[k][3] = in ? fv.at(x, y + 1) : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < (JC_P * JC_P + JC_THREADS - 1) / JC_THREADS; ++k) {
        const int i = threadIdx.x + k * JC_THREADS;
        if (i < JC_P * JC_P) {
            sp[0][i] = 0.0f;
            sp[1][i] = ring[k];
        }
    }
    __syncthreads();
    unsigned upd = 0, keep = 0;  // update cells; fully solid cells, which keep their value (every other one is 0)
    const float factor = U.dx * U.rho / U.dt;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = threadIdx.x + k * JC_THREADS, ly = i / JC_E, lx = i - ly * JC_E, x = x0 + lx, y = y0 + ly;
        const bool in = i < N && x >= 0 && y >= 0 && x < d.cx() && y < d.cy();
        const int at = in ? (ly + 1) * JC_P + lx + 1 : JC_P + 1;
        const float* l = sp[1] + at;
        const float lij = *l;
        const bool wet = in && !(lij >= 0.0f), open = !(w[k][0] == 0.0f && w[k][1] == 0.0f && w[k][2] == 0.0f && w[k][3] == 0.0f);
        const float nb[4] = {l[-1], l[1], l[-JC_P], l[JC_P]};
        float c = 0.0f, ww[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // fminf(0, nb / lij) is 0 unless nb > 0
            const float ff = wet && nb[q] > 0.0f ? fminf(0.0f, nb[q] / lij) : 0.0f;
            const float t = w[k][q] * (1.0f - ff);
            c = q ? c + t : t;
            ww[q] = w[k][q] * (ff >= 0.0f ? 1.0f : 0.0f);
        }
        if (wet && !open) keep |= 1u << k;
        const bool u = wet && open && !(fabsf(c) < 1.0e-6f);
        if (u) upd |= 1u << k;
        coef[k] = u ? c : 1.0f;
        rhs[k] = factor * rhs[k];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[k][q] = u ? ww[q] : 0.0f;
        if (in) sp[0][at] = pv[k];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * JC_P; i += JC_THREADS) {  // the second image's ring
        const int e = i / JC_P, q = i % JC_P;
        sp[1][e == 0 ? q : e == 1 ? (JC_P - 1) * JC_P + q : e == 2 ? q * JC_P : q * JC_P + JC_P - 1] = 0.0f;
    }
    __syncthreads();
    int at[PER], need[PER];  // a cell's place, and the iterations after which the owned cells still depend on it
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = threadIdx.x + k * JC_THREADS, ly = i / JC_E, lx = i - ly * JC_E;
        at[k] = (ly + 1) * JC_P + lx + 1;
        need[k] = i < N ? min(min(lx, JC_E - 1 - lx), min(ly, JC_E - 1 - ly)) : -1;
    }
#pragma unroll 1
    for (int it = 0; it < JC_K; ++it) {
        const float* a = sp[it & 1];
        float* b = sp[(it & 1) ^ 1];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (need[k] <= it) continue;  // a value of the rim: too far out to reach an owned cell
            const float* c = a + at[k];
            float n = w[k][0] * c[-1] + w[k][1] * c[1] + w[k][2] * c[-JC_P] + w[k][3] * c[JC_P] - rhs[k];
            if (!((upd >> k) & 1u)) n = 1.0f;
            const float v = div_any(n, coef[k]);
            b[at[k]] = (upd >> k) & 1u ? v : (keep >> k) & 1u ? c[0] : 0.0f;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < JC_T * JC_T; i += JC_THREADS) {
        const int lx = JC_K + i % JC_T, ly = JC_K + i / JC_T, x = x0 + lx, y = y0 + ly;
        if (x < d.cx() && y < d.cy()) p_out.at(x, y) = sp[JC_K & 1][(ly + 1) * JC_P + lx + 1];
    }
}

// solve_velocity_u.wgsl:15-47 / solve_velocity_v.wgsl:15-45
template <int COMP>
EFL_DEV void solve_velocity_at(const PF& out0, const PF& in1, const PF& solid, const PF& p0, const PF& ls0,
                               const PF& face_frac, const Uniform& U, const Dom& d) {
    int x = gx(), y = gy();
    if (COMP == 0 ? (x > d.nx || y >= d.xrows()) : (x >= d.ycols() || y > d.ny)) return;
    const float factor = U.dt / (U.dx * U.rho);
    float fr = (x < d.nx && y < d.ny) ? face_frac.ld(x, y) : 0.0f;
    if (fr == 0.0f) {
        out0.st(x, y, solid.ld(x, y));
        return;
    }
    const int ox = COMP == 0 ? 1 : 0, oy = COMP == 0 ? 0 : 1;
    float pij = p0.ld(x, y), pm = p0.ld(x - ox, y - oy);
    float lp = ls0.ld(x, y), lm = ls0.ld(x - ox, y - oy);
    if (lm >= 0.0f && lp < 0.0f) {
        pm = lm / lp * pij;
    } else if (lm < 0.0f && lp >= 0.0f) {
        pij = lp / lm * pm;
    } else if (COMP == 0 && lm >= 0.0f && lp >= 0.0f) {
        out0.st(x, y, 0.0f);
        return;
    }
    float val = in1.ld(x, y);
    out0.st(x, y, val - factor * (pij - pm));
}
// Both components in one launch over the larger of their grids (blockIdx.z: 0 = u, 1 = v).
__global__ void k_solve_velocity_uv(PF u0, PF u1, PF us, PF v0, PF v1, PF vs, PF p0, PF ls0, PF fu, PF fv, Uniform U,
                                    Dom d) {
    if (blockIdx.z == 0)
        solve_velocity_at<0>(u0, u1, us, p0, ls0, fu, U, d);
    else
        solve_velocity_at<1>(v0, v1, vs, p0, ls0, fv, U, d);
}

// initialize_{u,v}_valid + the 10 extrapolation sweeps of render_node.rs:540-608
// in ONE launch: blockIdx.z = component; each CTA owns a 32 x 32 tile of
// faces and holds it with a 10-face halo in shared memory (each sweep reads
// the valid flags of the previous one and only valid neighbours' velocities,
// so the result equals 10 global sweeps).  Writes the velocity, the flags
// after the tenth sweep (the "in" plane) and after the ninth (the "out"
// plane), as the per-sweep kernels leave them.
//
// Latency and issue bound it (a few CTAs on small grids, each a chain of 10
// sweeps).  A face turns valid once and its value is computed once, in that
// sweep: one warp runs the ten sweeps on the flags alone (a 64-bit word per
// image row, two rows per lane, neighbour rows by shuffles) and leaves the
// sweep in which each face turns valid, and the faces of each sweep as a list;
// then a sweep is one face per thread, its neighbours being valid if their
// sweep is an earlier one.  The form before it (byte flags, every face visited
// in every sweep by 256 threads with run-time row divisions) took 39 us at
// 64^2 and 48 us at 768 x 512.
//
// Faces outside the reference's dispatch (floor(n / 64) * 64 rows or columns,
// pipeline.rs:175-186) keep their velocity and both their flag planes; each
// sweep reads their flag from the plane that it reads.
constexpr int EX_T = 32, EX_H = 10, EX_E = EX_T + 2 * EX_H, EX_THREADS = 512;
struct ExtrapArgs {
    PF f[2];
    PI vin[2], vout[2];
    PF ls;
    const float2* range;  // per 32 x 32 cell tile of ls: (min, max)
    int rtx, rty;         // cell tiles per row / column
    int cw[2], ch[2];     // faces covered by the dispatch, per component
};
// (min, max) of the level set over each 32 x 32 tile of cells (one CTA per tile).
__global__ void __launch_bounds__(256) k_ls_tile_range(PF ls, float2* range, int rtx) {
    const int x0 = blockIdx.x * EX_T, y0 = blockIdx.y * EX_T;
    float lo = INFINITY, hi = -INFINITY;
    int nan = 0;  // a NaN makes the tile non-uniform below
    for (int i = threadIdx.x; i < EX_T * EX_T; i += 256) {
        const int x = x0 + (i & (EX_T - 1)), y = y0 + i / EX_T;
        if (x < ls.w && y < ls.h) {
            const float v = ls.at(x, y);
            lo = fminf(lo, v);
            hi = fmaxf(hi, v);
            nan |= v != v;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __shared__ float slo[8], shi[8];
    if ((threadIdx.x & 31) == 0) {
        slo[threadIdx.x >> 5] = lo;
        shi[threadIdx.x >> 5] = hi;
    }
    const int any_nan = __syncthreads_or(nan);
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) {
            lo = fminf(lo, slo[k]);
            hi = fmaxf(hi, shi[k]);
        }
        range[blockIdx.y * rtx + blockIdx.x] = any_nan ? make_float2(NAN, NAN) : make_float2(lo, hi);
    }
}
__global__ void __launch_bounds__(EX_THREADS) k_extrapolate_fused(ExtrapArgs a) {
    typedef unsigned long long row_t;
    static_assert(EX_E <= 64 && EX_THREADS % 64 == 0 && EX_THREADS >= 320, "an image row is one word; two warps cover a row");
    constexpr int LW = EX_E + 2, NLS = LW * LW, NFC = EX_E * EX_E, PERF = (NFC + EX_THREADS - 1) / EX_THREADS;
    constexpr unsigned char NEVER = 15, OUTSIDE = 16;
    __shared__ float sf[NFC];
    __shared__ float sl[NLS];          // level set of the cells (x0 - 1 .., y0 - 1 ..)
    __shared__ row_t sv[64];           // valid flags at the start, bit lx
    __shared__ row_t stat[2][64];      // flags of the faces outside the dispatch, "in" and "out" plane
    __shared__ row_t fresh_s[10][64];  // faces that turn valid in a sweep
    __shared__ unsigned char st[NFC];  // 1 + the sweep in which a face turns valid (0: at the start, NEVER: not in
                                       // ten sweeps); OUTSIDE + both flags of a face outside the dispatch
    __shared__ unsigned short list[NFC];
    __shared__ int total, first_of[10], count_of[10];
    const int comp = blockIdx.z;
    const PF f = a.f[comp];
    const PI vin = a.vin[comp], vout = a.vout[comp];
    const int W = f.w, H = f.h, CW = a.cw[comp], CH = a.ch[comp];
    const int x0 = blockIdx.x * EX_T - EX_H, y0 = blockIdx.y * EX_T - EX_H;
    const int tid = threadIdx.x;
    // The same flag for every owned face.
    auto write_flags = [&](int v) {
        for (int i = tid; i < EX_T * EX_T / 4; i += EX_THREADS) {
            const int x = x0 + EX_H + (i & 7) * 4, y = y0 + EX_H + (i >> 3);
            if (y >= CH) continue;
            if (x + 3 < CW) {  // x is a multiple of 4 and the pitch one of 32: 16-byte aligned
                *reinterpret_cast<int4*>(&vin.at(x, y)) = make_int4(v, v, v, v);
                *reinterpret_cast<int4*>(&vout.at(x, y)) = make_int4(v, v, v, v);
            } else {
                for (int k = x; k < CW; ++k) vin.at(k, y) = vout.at(k, y) = v;
            }
        }
    };
    const bool covered = min(x0 + EX_E, W) <= CW && min(y0 + EX_E, H) <= CH;
    // Every face the tile's image and flags read lies over the 3 x 3 cell tiles around it (the 10-face halo
    // and the one-cell level-set stencil stay within one tile).  All of their level set < 0: every face is
    // valid (area_fraction <= 0); all of it > 1e-30: none is (area_fraction > 0; the bound keeps the corner
    // averages normal).  Either way the ten sweeps change nothing: write the flags only.
    if (covered) {
        int neg = 1, pos = 1;
        if (tid < 9) {
            const int tx = min(max((int)blockIdx.x - 1 + tid % 3, 0), a.rtx - 1);
            const int ty = min(max((int)blockIdx.y - 1 + tid / 3, 0), a.rty - 1);
            const float2 r = a.range[ty * a.rtx + tx];
            neg = r.y < 0.0f;    // false for NaN
            pos = r.x > 1e-30f;  // false for NaN
        }
        const int all_neg = __syncthreads_and(neg), all_pos = __syncthreads_and(pos);
        if (all_neg || all_pos) {
            write_flags(all_neg ? 1 : 0);
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < (NLS + EX_THREADS - 1) / EX_THREADS; ++k) {
        const int i = tid + k * EX_THREADS;
        if (i < NLS) sl[i] = a.ls.ld(x0 - 1 + i % LW, y0 - 1 + i / LW);
    }
#pragma unroll
    for (int k = 0; k < PERF; ++k) {
        const int i = tid + k * EX_THREADS;
        if (i < NFC) sf[i] = f.ld(x0 + i % EX_E, y0 + i / EX_E);
    }
    if (tid < 64) sv[tid] = stat[0][tid] = stat[1][tid] = 0;
    if (tid == 0) total = 0;
    __syncthreads();
    // Two warps per image row: lane = column, the second warp 32 columns on.
    const int lane = tid & 31, half = (tid >> 5) & 1, row0 = tid >> 6;
    constexpr int ROWS = EX_THREADS / 64, PER = (EX_E + ROWS - 1) / ROWS;
    const int lx = half * 32 + lane, x = x0 + lx;
    int any_valid = 0, any_invalid = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int ly = row0 + k * ROWS, y = y0 + ly;
        if (ly >= EX_E) break;
        bool v = false, s0 = false, s1 = false;
        if (lx < EX_E && (unsigned)x < (unsigned)W && (unsigned)y < (unsigned)H) {
            if (x < CW && y < CH) {
                // extrapolate/initialize_{u,v}_valid.wgsl; c[LW + 1] is the cell (x, y)
                const float* c = sl + ly * LW + lx;
                const float c0 = c[0], c3 = c[LW + 1];
                const float c1 = comp == 0 ? c[1] : c[LW], c2 = comp == 0 ? c[LW] : c[1];
                const float c4 = comp == 0 ? c[2 * LW] : c[2], c5 = comp == 0 ? c[2 * LW + 1] : c[LW + 2];
                const float vm = 0.25f * (c0 + c1 + c2 + c3);
                const float vp = 0.25f * (c2 + c3 + c4 + c5);
                v = !area_fraction_positive(vm, vp);
            } else {
                s0 = vin.at(x, y) == 1;
                s1 = vout.at(x, y) == 1;
                v = s0;
            }
            if (v) any_valid = 1;
            else any_invalid = 1;
            if (s0 != s1) any_valid = any_invalid = 1;
        }
        const unsigned b = __ballot_sync(0xffffffffu, v);
        if (lane == 0) reinterpret_cast<unsigned*>(&sv[ly])[half] = b;
        if (!covered) {
            const unsigned b0 = __ballot_sync(0xffffffffu, s0), b1 = __ballot_sync(0xffffffffu, s1);
            if (lane == 0) {
                reinterpret_cast<unsigned*>(&stat[0][ly])[half] = b0;
                reinterpret_cast<unsigned*>(&stat[1][ly])[half] = b1;
            }
        }
    }
    // A tile whose image is all valid or all invalid comes out of the ten sweeps unchanged, with both flag
    // planes equal to the start flag (only faces inside the domain count).
    const int has_valid = __syncthreads_or(any_valid), has_invalid = __syncthreads_or(any_invalid);
    if (!(has_valid && has_invalid)) {
        write_flags(has_valid ? 1 : 0);
        return;
    }
    // The sweeps on the flags (extrapolate_{u,v}.wgsl:5-63): lane l holds the image rows 2 l and 2 l + 1.
    if (tid < 32) {
        auto cols = [&](int lo, int hi) -> row_t {  // the columns whose x lies in [lo, hi)
            const int l = max(lo - x0, 0), h = min(hi - x0, EX_E);
            return l >= h ? 0ull : ((1ull << (h - l)) - 1ull) << l;
        };
        const row_t mcov = cols(0, CW), mright = cols(0, W - 1), mleft = cols(2, W), mup = cols(1, W);
        row_t v[2], s0[2], s1[2], mc[2], ml[2], mu[2], md[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int ly = 2 * tid + q, y = y0 + ly;
            v[q] = sv[ly];
            s0[q] = covered ? 0 : stat[0][ly];
            s1[q] = covered ? 0 : stat[1][ly];
            mc[q] = y >= 0 && y < CH && ly < EX_E ? mcov : 0;
            ml[q] = y > 0 ? mleft : 0;
            md[q] = y + 1 < H ? ~0ull : 0;
            mu[q] = y - 1 > 0 ? mup : 0;
        }
        for (int s = 0; s < 10; ++s) {
            row_t up = __shfl_up_sync(0xffffffffu, v[1], 1), dn = __shfl_down_sync(0xffffffffu, v[0], 1);
            if (tid == 0) up = 0;
            if (tid == 31) dn = 0;
            const row_t n0 = ((v[0] >> 1) & mright) | ((v[0] << 1) & ml[0]) | (v[1] & md[0]) | (up & mu[0]);
            const row_t n1 = ((v[1] >> 1) & mright) | ((v[1] << 1) & ml[1]) | (dn & md[1]) | (v[0] & mu[1]);
            const row_t f0 = ~v[0] & n0 & mc[0], f1 = ~v[1] & n1 & mc[1];
            fresh_s[s][2 * tid] = f0;
            fresh_s[s][2 * tid + 1] = f1;
            v[0] = (v[0] & mc[0]) | f0 | (s & 1 ? s0[0] : s1[0]);  // as the next sweep reads them
            v[1] = (v[1] & mc[1]) | f1 | (s & 1 ? s0[1] : s1[1]);
        }
    }
    if (tid >= 32) {  // meanwhile: the faces that never turn valid so far, the valid ones, the ones outside
        for (int i = tid - 32; i < NFC; i += EX_THREADS - 32) {
            const int ly = i / EX_E, c = i - ly * EX_E;
            int n = (sv[ly] >> c) & 1ull ? 0 : NEVER;
            if (!covered && (x0 + c >= CW || y0 + ly >= CH))
                n = OUTSIDE + (int)((stat[0][ly] >> c) & 1ull) + 2 * (int)((stat[1][ly] >> c) & 1ull);
            st[i] = (unsigned char)n;
        }
    }
    __syncthreads();
    // The faces of each sweep as a list (a warp per sweep, two rows per lane).
    if (tid < 320) {
        const int s = tid >> 5;
        row_t f[2] = {fresh_s[s][2 * lane], fresh_s[s][2 * lane + 1]};
        const int n = __popcll(f[0]) + __popcll(f[1]);
        int pre = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += q;
        }
        int base = 0;
        if (lane == 31) {
            base = pre ? atomicAdd(&total, pre) : 0;
            first_of[s] = base;
            count_of[s] = pre;
        }
        int to = __shfl_sync(0xffffffffu, base, 31) + pre - n;
#pragma unroll
        for (int q = 0; q < 2; ++q)
            for (row_t m = f[q]; m; m &= m - 1) {
                const int i = (2 * lane + q) * EX_E + __ffsll(m) - 1;
                list[to++] = (unsigned short)i;
                st[i] = (unsigned char)(s + 1);
            }
    }
    __syncthreads();
    for (int s = 0; s < 10; ++s) {
        for (int j = tid; j < count_of[s]; j += EX_THREADS) {
            const int i = list[first_of[s] + j], ly = i / EX_E, c = i - ly * EX_E, gx = x0 + c, gy = y0 + ly;
            // Every load first; a face on the image's rim misses a neighbour, and its value is not read by the
            // faces the tile owns.
            const int r = min(i + 1, NFC - 1), l = max(i - 1, 0), dn = min(i + EX_E, NFC - 1), up = max(i - EX_E, 0);
            auto valid = [&](int n) -> bool { return n < OUTSIDE ? n <= s : (n >> (s & 1)) & 1; };
            const bool vr = gx + 1 < W && c + 1 < EX_E && valid(st[r]), vl = gx - 1 > 0 && gy > 0 && c > 0 && valid(st[l]);
            const bool vd = gy + 1 < H && ly + 1 < EX_E && valid(st[dn]);
            const bool vu = gx > 0 && gy - 1 > 0 && ly > 0 && valid(st[up]);
            const float fr = sf[r], fl = sf[l], fd = sf[dn], fu = sf[up];
            float nu = 0.0f;  // neighbour order and bounds as the reference
            nu = vr ? nu + fr : nu;
            nu = vl ? nu + fl : nu;
            nu = vd ? nu + fd : nu;
            nu = vu ? nu + fu : nu;
            sf[i] = nu / (float)((int)vr + (int)vl + (int)vd + (int)vu);
        }
        __syncthreads();
    }
    for (int i = tid; i < EX_T * EX_T; i += EX_THREADS) {
        const int oy = EX_H + i / EX_T, ox = EX_H + i % EX_T, gx = x0 + ox, gy = y0 + oy;
        if (gx >= CW || gy >= CH) continue;
        f.at(gx, gy) = sf[oy * EX_E + ox];
        vin.at(gx, gy) = st[oy * EX_E + ox] <= 10;  // after the tenth sweep
        vout.at(gx, gy) = st[oy * EX_E + ox] <= 9;  // after the ninth
    }
}

// advect_levelset.wgsl:49-74
EFL_DEV float cubic1d(float y0, float y1, float y2, float y3, float t) {
    float d1 = 0.5f * (y2 - y0);
    float d2 = 0.5f * (y3 - y1);
    float a0 = y1, a1 = d1;
    float a2 = -2.0f * d1 - d2 + 3.0f * (y2 - y1);
    float a3 = d1 + d2 - 2.0f * (y2 - y1);
    return a3 * t * t * t + a2 * t * t + a1 * t + a0;
}
EFL_DEV float cubic1d_x(const PF& t, int bx, int by, float tx) {
    return cubic1d(t.ld(bx - 1, by), t.ld(bx, by), t.ld(bx + 1, by), t.ld(bx + 2, by), tx);
}
// advect_levelset.wgsl:11-34 (CUBIC defined, advect_levelset.rs:62)
EFL_DEV float advected_level(const PF& u0, const PF& v0, const PF& ls0, float dt, const Dom& d, int x, int y) {
    float2 xn = runge_kutta(u0, v0, (float)x, (float)y, dt);
    xn.x = fclampf(xn.x, 0.0f, (float)d.nx - 1.0f);
    xn.y = fclampf(xn.y, 0.0f, (float)d.ny - 1.0f);
    int bx = f2i(xn.x), by = f2i(xn.y);
    float tx = xn.x - (float)bx, ty = xn.y - (float)by;
    float r[4];
    if (bx >= 1 && by >= 1 && bx + 2 < d.nx && by + 2 < d.ny) {  // one test for the interior
        const float* c = ls0.p + (size_t)(by - 1) * ls0.P + bx;
#pragma unroll
        for (int k = 0; k < 4; ++k, c += ls0.P) r[k] = cubic1d(c[-1], c[0], c[1], c[2], tx);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = cubic1d_x(ls0, bx, by - 1 + k, tx);
    }
    return cubic1d(r[0], r[1], r[2], r[3], ty);
}
__global__ void k_advect_levelset(PF u0, PF v0, PF ls0, PF ls1, float dt, Dom d) {
    const int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    const float nl = advected_level(u0, v0, ls0, dt, d, x, y);
    if (fabsf(nl) < 1000.0f) ls1.st(x, y, nl);
}

// update_fluid_source.wgsl:72-107
struct Sources {
    efl_source s[EFL_MAX_FLUID_SOURCE];
    int n;
};
EFL_DEV float level_aabb(float hx, float hy, float cx, float cy, float px, float py) {
    float dx = fabsf(cx - px) - hx, dy = fabsf(cy - py) - hy;
    bool ix = dx < 0.0f, iy = dy < 0.0f;
    if (ix) return iy ? fmaxf(dx, dy) : dy;
    return iy ? dx : wlength(dx, dy);
}
EFL_DEV float level_source(const efl_source& s, float px, float py) {
    switch (s.shape) {
        case EFL_SOURCE_CIRCLE: return wlength(s.center[0] - px, s.center[1] - py) - s.data[0];
        case EFL_SOURCE_AABB: return level_aabb(s.data[0], s.data[1], s.center[0], s.center[1], px, py);
        default: return 0.0f;
    }
}
// update_fluid_source.wgsl:30-62: level set and per-cell source velocity.
__global__ void k_fluid_source_cells(PF ls1, PU upd, P2 vel, Sources S, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    const float dimx = (float)d.nx, dimy = (float)d.ny;
    float uvx = (float)(uint32_t)x / dimx, uvy = (float)(uint32_t)y / dimy;
    float ndcx = uvx * 2.0f + -1.0f, ndcy = uvy * -2.0f + 1.0f;  // bevy uv_to_ndc
    float px = 0.5f * dimx * ndcx, py = 0.5f * dimy * ndcy;
    float nl = ls1.ld(x, y);
    float vx = 0.0f, vy = 0.0f;
    bool has_source = false, vu = false;
    for (int i = 0; i < S.n; ++i) {
        const efl_source& src = S.s[i];
        float sdf = level_source(src, px, py);
        if (src.mode == EFL_SOURCE_MODE_SOURCE) {
            nl = fminf(nl, sdf);
            has_source = true;
            if (sdf < 0.0f) {
                vx = vx + src.velocity[0];
                vy = vy + src.velocity[1];
                vu = true;
            }
        } else if (!has_source) {
            nl = fmaxf(nl, -sdf);
        }
    }
    ls1.st(x, y, nl);
    upd.st(x, y, vu ? 1u : 0u);
    vel.st(x, y, make_float2(vx, vy));
}
// update_fluid_source.wgsl:64-69: a face written by two invocations takes
// the raster-last writer's value (the cell on its high side).
__global__ void k_fluid_source_faces(PF u0, PF v0, PU upd, P2 vel, Dom d) {
    int x = gx(), y = gy();
    const int W = d.cx(), H = d.cy();
    if (x <= W && y < H) {  // u face (x, y): writers (x, y) then (x-1, y)
        if (x < W && upd.ld(x, y)) u0.st(x, y, vel.ld(x, y).x);
        else if (x >= 1 && upd.ld(x - 1, y)) u0.st(x, y, vel.ld(x - 1, y).x);
    }
    if (x < W && y <= H) {  // v face (x, y): writers (x, y) then (x, y-1)
        if (y < H && upd.ld(x, y)) v0.st(x, y, vel.ld(x, y).y);
        else if (y >= 1 && upd.ld(x, y - 1)) v0.st(x, y, vel.ld(x, y - 1).y);
    }
}

// jump_flooding/initialize.wgsl:8-41
__global__ void k_jfa_init(PF ls1, P2 seeds, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    float md = 10.0f;
    float2 seed = make_float2(-1.0f, -1.0f);
    float level = ls1.ld(x, y);
    for (int i = -1; i <= 1; ++i)
        for (int j = -1; j <= 1; ++j) {
            if (i == 0 && j == 0) continue;
            int ax = x + i, ay = y + j;
            if (ax < 0 || ay < 0 || ax >= d.nx || ay >= d.ny) continue;
            float nl = ls1.ld(ax, ay);
            if (nl >= 0.0f && !(level >= 0.0f)) {
                float t = level / (level - nl);
                if (fabsf(t) < md) {
                    md = fabsf(t);
                    seed = make_float2((float)x + t * (float)i, (float)y + t * (float)j);
                }
            }
        }
    seeds.st(x, y, seed);
}
EFL_DEV bool valid_seed(float2 s) { return s.x != -1.0f && s.y != -1.0f; }
// jump_flooding/iterate.wgsl:18-56
__global__ void k_jfa_iterate(P2 in, P2 out, int step, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    float2 cur = in.ld(x, y), best = cur;
    float bd = 1e10f;
    if (valid_seed(cur)) bd = wlength(cur.x - (float)x, cur.y - (float)y);
    for (int i = -1; i <= 1; ++i)
        for (int j = -1; j <= 1; ++j) {
            if (i == 0 && j == 0) continue;
            int ax = x + i * step, ay = y + j * step;
            if (ax < 0 || ay < 0 || ax >= in.w || ay >= in.h) continue;
            float2 ns = in.at(ax, ay);
            if (!valid_seed(ns)) continue;
            float cd = wlength(ns.x - (float)x, ns.y - (float)y);
            if (cd < bd) {
                best = ns;
                bd = cd;
            }
        }
    out.st(x, y, best);
}
// jump_flooding/calculate_sdf.wgsl:9-23
__global__ void k_jfa_sdf(P2 seeds, PF ls1, PF ls0, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    float2 s = seeds.ld(x, y);
    float sdf = wlength(s.x - (float)x, s.y - (float)y);
    float level = ls1.ld(x, y);
    ls0.st(x, y, sdf * (level < 0.0f ? -1.0f : 1.0f));
}

// fast_iterative_method/update.wgsl:13-54 in its deterministic two-phase form (the reference writes neighbours
// from inside one dispatch, a data race), together with initialize.wgsl:10-40 and
// initialize_active_label.wgsl:8-40, in ONE launch per FIM_HALO / 2 iterations.  Phase A: active cells update
// from the iteration-start phi and flag convergence.  Phase B: an inactive cell next to a cell that converged
// in A is re-solved from the post-A phi and activated, with the sign of the raster-last converged neighbour
// (down, right, left, up).
//
// A CTA owns FIM_TW x FIM_TH cells and holds them with a halo of FIM_HALO cells in shared memory.  One
// iteration's result at a cell depends on cells at most 2 away (phase A reads radius 1, phase B reads phase A's
// result at radius 1), so values go wrong only near the image's edge, 2 cells deeper per iteration: after
// FIM_HALO / 2 iterations the owned cells are exact.  INIT: the start state comes from the advected level set
// (source cells, sign * large elsewhere, active neighbours of the sources); otherwise from the planes (S, L) of
// the launch before, which must be another pair than (SD, LD): a CTA that starts late must still see its
// neighbours' values of the launch's start.
//
// The cells that change form a thin band around the interface, and on small grids the work is latency- and
// issue-bound (a few CTAs and a chain of 10 iterations).  So the CTA keeps the active cells as a list in shared
// memory, one cell per thread, and the labels as bit masks, one word per 32 columns of an image row, one word per
// thread: phase A solves the listed cells and marks those that converged, the words beside converged cells give
// the candidates of phase B (each once, whatever the number of its converged neighbours), and phase B solves the
// listed candidates.  The images s and t differ at active cells alone: A writes t there, B copies those back and
// writes s where it activates, and A rewrites t at every active cell before B reads it.  The order of a list does
// not matter: a phase reads one image and writes the other.
// The start state costs no launch of its own.  Before: two launches for the start state, then 20 per-phase
// launches (2.0 + 3.0 us each at 256^2) or, on large grids, a 72 x 72 image with every cell visited in every
// phase (181 us at 2048^2, 379 us at 4096^2).
constexpr int FIM_HALO = 20, FIM_TW = 56, FIM_TH = 32, FIM_THREADS = 768;
constexpr int FIM_IW = FIM_TW + 2 * FIM_HALO, FIM_IH = FIM_TH + 2 * FIM_HALO, FIM_NW = FIM_IW / 32;
constexpr int FIM_PW = FIM_IW + 2;                        // row pitch of s and t: a ring of large values
constexpr int FIM_LW = FIM_IW + 4, FIM_LH = FIM_IH + 4;   // staged level set: the image and two cells around it
constexpr int FIM_CELLS = ((FIM_IH + 2) * FIM_PW + 3) / 4 * 4;
constexpr int FIM_TBUF = FIM_CELLS > FIM_LW * FIM_LH ? FIM_CELLS : FIM_LW * FIM_LH;
constexpr int FIM_WORDS = FIM_IH * FIM_NW, FIM_LIST = FIM_IW * FIM_IH;
typedef unsigned FimMask[FIM_IH + 2][FIM_NW + 2];  // [row + 1][word + 1]: a rim of zeros
struct FimTile {
    float s[FIM_CELLS], t[FIM_TBUF];  // t: the staged level set first
    FimMask src, act, conv[2];        // source, active (converged ones included), converged in even / odd iterations
    int count[2], ncand;
    unsigned short list[2][FIM_LIST], cand[FIM_LIST];
};
constexpr size_t FIM_SMEM = sizeof(FimTile);
// update.wgsl:56-83 on an image with a ring of large values (abs_get_phi gives that outside the domain)
EFL_DEV float fim_solve(const float* a, int i) {
    const float xm = fminf(fabsf(a[i - 1]), fabsf(a[i + 1]));
    const float ym = fminf(fabsf(a[i - FIM_PW]), fabsf(a[i + FIM_PW]));
    const float d = xm - ym;
    const bool one = d > SQRT2_F || d < -SQRT2_F;  // from one side only (selects: no divergent chains)
    const float both = 0.5f * (xm + ym + sqrtf(one ? 1.0f : 2.0f - d * d));
    return one ? (d > SQRT2_F ? ym : xm) + 1.0f : both;
}
// Appends i to list for the lanes with `take` (a whole warp calls it).
EFL_DEV void fim_append(unsigned short* list, int* count, bool take, int i) {
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
    int at = 0;
    if (lane == lead) at = atomicAdd(count, __popc(m));
    at = __shfl_sync(0xffffffffu, at, lead);
    if (take) list[at + __popc(m & ((1u << lane) - 1u))] = (unsigned short)i;
}
template <bool INIT>
__global__ void __launch_bounds__(FIM_THREADS, 2) k_fim(PF S, PU L, PF SD, PU LD, Dom d, int iters, int tiles_x) {
    static_assert(FIM_IW % 32 == 0 && 2 * FIM_WORDS <= FIM_THREADS && 2 * (FIM_IH + 2) <= FIM_THREADS,
                  "image rows of whole words, two threads per word, one per rim cell");
    extern __shared__ __align__(16) unsigned char fim_raw[];
    FimTile& T = *reinterpret_cast<FimTile*>(fim_raw);
    float *s = T.s, *t = T.t;
    constexpr int WARPS = FIM_THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x0 = (int)(blockIdx.x % tiles_x) * FIM_TW - FIM_HALO, y0 = (int)(blockIdx.x / tiles_x) * FIM_TH - FIM_HALO;
    const int W = d.nx, H = d.ny;  // the dispatch domain (sizes are multiples of 8) and the planes' extent
    for (int i = tid; i < 4 * (int)(sizeof(FimMask) / 4); i += FIM_THREADS) (&T.src[0][0])[i] = 0u;
    if (tid < 2) T.count[tid] = 0;
    // The ring of s.
    for (int i = tid; i < 2 * FIM_PW + 2 * FIM_IH; i += FIM_THREADS) {
        const int at = i < FIM_PW       ? i
                       : i < 2 * FIM_PW ? (FIM_IH + 1) * FIM_PW + i - FIM_PW
                                        : ((i - 2 * FIM_PW) / 2 + 1) * FIM_PW + (i & 1) * (FIM_PW - 1);
        s[at] = FIM_LARGE;
    }
    if constexpr (INIT) {
        // The level set, NaN outside the domain: no product with it is <= 0.
#pragma unroll
        for (int k = 0; k < (FIM_LW * FIM_LH + FIM_THREADS - 1) / FIM_THREADS; ++k) {
            const int i = tid + k * FIM_THREADS, gx = x0 - 2 + i % FIM_LW, gy = y0 - 2 + i / FIM_LW;
            if (i < FIM_LW * FIM_LH)
                t[i] = (unsigned)gx < (unsigned)W && (unsigned)gy < (unsigned)H ? S.at(gx, gy) : NAN;
        }
        __syncthreads();
        // initialize.wgsl: a source cell has an in-domain neighbour of another sign (or is 0)
        auto source = [&](const float* q) -> bool {
            const float l = *q;
            return (l * q[-1] <= 0.0f) | (l * q[1] <= 0.0f) | (l * q[-FIM_LW] <= 0.0f) | (l * q[FIM_LW] <= 0.0f);
        };
#pragma unroll 5
        for (int it = warp; it < (FIM_IH + 2) * FIM_NW; it += WARPS) {
            const int r = it / FIM_NW, w = it % FIM_NW, ix = 32 * w + lane;  // image row r - 1
            const float* q = t + (r + 1) * FIM_LW + ix + 2;
            const bool sc = source(q);
            const unsigned b = __ballot_sync(0xffffffffu, sc);
            if (lane == 0) T.src[r][w + 1] = b;
            if (r >= 1 && r <= FIM_IH) {
                const bool in = (unsigned)(x0 + ix) < (unsigned)W && (unsigned)(y0 + r - 1) < (unsigned)H;
                s[r * FIM_PW + ix + 1] = in ? (sc ? *q : wsign(*q) * FIM_LARGE) : FIM_LARGE;
            }
        }
        if (tid < 2 * (FIM_IH + 2)) {  // the cells beside the image's first and last column
            const int r = tid >> 1;
            if (tid & 1) T.src[r][FIM_NW + 1] = source(t + (r + 1) * FIM_LW + FIM_IW + 2) ? 1u : 0u;
            else T.src[r][0] = source(t + (r + 1) * FIM_LW + 1) ? 0x80000000u : 0u;
        }
    } else {
        for (int it = warp; it < FIM_WORDS; it += WARPS) {
            const int r = it / FIM_NW + 1, w = it % FIM_NW, gx = x0 + 32 * w + lane, gy = y0 + r - 1;
            uint32_t l = LABEL_NONE;
            float v = FIM_LARGE;
            if ((unsigned)gx < (unsigned)W && (unsigned)gy < (unsigned)H) {
                l = L.at(gx, gy);
                v = S.at(gx, gy);
            }
            s[r * FIM_PW + 32 * w + lane + 1] = v;
            const unsigned b = __ballot_sync(0xffffffffu, l == LABEL_SOURCE);
            const unsigned a = __ballot_sync(0xffffffffu, l == LABEL_ACTIVE);
            if (lane == 0) {
                T.src[r][w + 1] = b;
                T.act[r][w + 1] = a;
            }
        }
    }
    __syncthreads();
    // This thread's half of a word (the cells of a word are listed by two threads): the cells in the domain, and
    // (row, word) of the masks.
    const int wi = tid >> 1, mr = min(wi / FIM_NW, FIM_IH - 1) + 1, mw = wi % FIM_NW + 1;
    const unsigned mine = tid & 1 ? 0xffff0000u : 0xffffu;
    const int wx = x0 + 32 * (mw - 1), cell0 = mr * FIM_PW + 32 * (mw - 1) + 1;
    const bool word = wi < FIM_WORDS && y0 + mr - 1 >= 0 && y0 + mr - 1 < H;
    const unsigned dom = !word || wx >= W || wx <= -32
                             ? 0u
                             : (W - wx >= 32 ? ~0u : (1u << (W - wx)) - 1u) & (wx >= 0 ? ~0u : ~0u << -wx);
    // Lists the cells of bits m, the word's; cells of one word stay together.
    auto list_bits = [&](unsigned short* list, int* count, unsigned m) {
        if (!m) return;
        int at = atomicAdd(count, __popc(m));
        for (; m; m &= m - 1) list[at++] = (unsigned short)(cell0 + __ffs(m) - 1);
    };
    auto beside = [&](const FimMask& M) -> unsigned {  // the word's cells with a marked neighbour
        const unsigned c = M[mr][mw];
        return M[mr + 1][mw] | M[mr - 1][mw] | (c >> 1) | (M[mr][mw + 1] << 31) | (c << 1) | (M[mr][mw - 1] >> 31);
    };
    if (word) {
        // initialize_active_label.wgsl: every other in-domain cell beside a source cell
        const unsigned a = INIT ? beside(T.src) & ~T.src[mr][mw] & dom : T.act[mr][mw];
        if (INIT && (tid & 1)) T.act[mr][mw] = a;
        list_bits(T.list[0], &T.count[0], a & mine);
    }
    __syncthreads();
    // A cell changes only while it is active, so an image without an active cell (most of a large grid) stays.
    int n = T.count[0];
    if (n) {
        for (int i = tid; i < FIM_CELLS / 4; i += FIM_THREADS)
            reinterpret_cast<float4*>(t)[i] = reinterpret_cast<const float4*>(s)[i];
        __syncthreads();
        for (int k = 0; k < iters; ++k) {
            const int cur = k & 1, nxt = cur ^ 1;
            FimMask& conv = T.conv[cur];
            // phase A
            for (int j = tid; j < (n + 31) / 32 * 32; j += FIM_THREADS) {
                bool still = false;
                int i = 0;
                if (j < n) {
                    i = T.list[cur][j];
                    const float p = s[i];
                    const float q = fim_solve(s, i) * wsign(p);
                    t[i] = q;
                    still = fabsf(p - q) > FIM_EPS;
                    if (!still) {
                        const int r = i / FIM_PW, x = i - r * FIM_PW - 1;
                        atomicOr(&conv[r][(x >> 5) + 1], 1u << (x & 31));
                    }
                }
                fim_append(T.list[nxt], &T.count[nxt], still, i);
            }
            if (tid == 0) T.ncand = 0;
            __syncthreads();
            // phase B: inactive cells beside a converged one
            if (word) {
                const unsigned a = T.act[mr][mw];
                list_bits(T.cand, &T.ncand, beside(conv) & ~(a | T.src[mr][mw]) & dom & mine);
            }
            for (int j = tid; j < n; j += FIM_THREADS) {
                const int i = T.list[cur][j];
                s[i] = t[i];
            }
            __syncthreads();
            const int nc = T.ncand;
            if (word && (tid & 1)) atomicAnd(&T.act[mr][mw], ~conv[mr][mw]);  // free again
            for (int j = tid; j < (nc + 31) / 32 * 32; j += FIM_THREADS) {
                bool fresh = false;
                int c = 0;
                if (j < nc) {
                    c = T.cand[j];
                    const float qn = fim_solve(t, c);
                    if (fabsf(t[c]) > qn) {
                        const int r = c / FIM_PW, x = c - r * FIM_PW - 1, w = (x >> 5) + 1, b = x & 31;
                        const unsigned right = (conv[r][w] >> 1) | (conv[r][w + 1] << 31);
                        const unsigned left = (conv[r][w] << 1) | (conv[r][w - 1] >> 31);
                        const int from = (conv[r + 1][w] >> b) & 1u ? c + FIM_PW
                                         : (right >> b) & 1u        ? c + 1
                                         : (left >> b) & 1u         ? c - 1
                                                                    : c - FIM_PW;
                        s[c] = qn * wsign(t[from]);
                        atomicOr(&T.act[r][w], 1u << b);
                        fresh = true;
                    }
                }
                fim_append(T.list[nxt], &T.count[nxt], fresh, c);
            }
            if (tid < FIM_WORDS) T.conv[nxt][tid / FIM_NW + 1][tid % FIM_NW + 1] = 0u;
            if (tid == 0) T.count[cur] = 0;
            __syncthreads();
            n = T.count[nxt];
        }
    }
    for (int i = tid; i < FIM_TW * FIM_TH; i += FIM_THREADS) {
        const int ix = FIM_HALO + i % FIM_TW, iy = FIM_HALO + i / FIM_TW;
        const int gx = x0 + ix, gy = y0 + iy;
        if (gx < W && gy < H) {
            const int w = (ix >> 5) + 1, b = ix & 31;
            SD.at(gx, gy) = s[(iy + 1) * FIM_PW + ix + 1];
            LD.at(gx, gy) = (T.src[iy + 1][w] >> b) & 1u   ? LABEL_SOURCE
                            : (T.act[iy + 1][w] >> b) & 1u ? LABEL_ACTIVE
                                                           : LABEL_NONE;
        }
    }
}

// levelset_gradient.wgsl:4-21
__global__ void k_gradient(PF ls0, P2 grad, Dom d) {
    int x = gx(), y = gy();
    if (x >= d.cx() || y >= d.cy()) return;
    if (x == 0 || y == 0 || x >= d.nx || y >= d.ny) return;
    grad.st(x, y, make_float2(0.5f * (ls0.ld(x + 1, y) - ls0.ld(x - 1, y)), 0.5f * (ls0.ld(x, y + 1) - ls0.ld(x, y - 1))));
}

// solid_obstacle.wgsl:67-89
EFL_DEV float2 center_of_mass(const efl_solid_obstacle& o) {
    switch (o.shape) {
        case EFL_SHAPE_CIRCLE:
        case EFL_SHAPE_RECTANGLE:
        case EFL_SHAPE_CAPSULE:
            return make_float2(o.transform[12], o.transform[13]);
        case EFL_SHAPE_TRIANGLE: {
            float lx = (o.values[0] + o.values[2] + o.values[4]) / 3.0f;
            float ly = (o.values[1] + o.values[3] + o.values[5]) / 3.0f;
            return mat_xy(o.transform, lx, ly);
        }
        default:
            return make_float2(0.0f, 0.0f);
    }
}
// sample_forces.wgsl:20-53.  Per-cell force/torque in fixed point
// (fixed_point_conversion.wgsl:2-13, scale 0.1 -> x10), accumulated in a
// block-private shared-memory copy of the 3 x 256 bins and flushed with
// one global atomic per touched bin.  Integer sums are order-independent,
// so the bins are bit-identical to the reference's per-cell atomics.
__global__ void k_solid_forces(PF fu, PF fv, PI sid, PF p0, const efl_solid_obstacle* __restrict__ obs, int n_obs,
                               Uniform U, Dom d, int* __restrict__ bins) {
    __shared__ int sb[3 * EFL_MAX_SOLIDS];
    __shared__ int touched;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int nth = blockDim.x * blockDim.y;
    for (int i = tid; i < 3 * EFL_MAX_SOLIDS; i += nth) sb[i] = 0;
    if (tid == 0) touched = 0;
    __syncthreads();
    int x = gx(), y = gy();
    if (x < d.cx() && y < d.cy()) {
        float f0 = fu.at(x, y), f1 = fu.at(x + 1, y), f2 = fv.at(x, y), f3 = fv.at(x, y + 1);
        int32_t id = sid.at(x, y);
        if (!(f0 == 0.0f && f1 == 0.0f && f2 == 0.0f && f3 == 0.0f) && id != -1) {
            float p = p0.at(x, y);
            float fx = -(f1 - f0) * p * U.dx;
            float fy = -(f3 - f2) * p * U.dx;
            float2 c = make_float2(0.0f, 0.0f);
            if (id >= 0 && id < n_obs) c = center_of_mass(obs[id]);
            float uvx = (float)x / U.size[0], uvy = (float)y / U.size[1];
            float xx = (uvx - 0.5f) * U.size[0], yy = (-uvy + 0.5f) * U.size[1];
            float2 w = mat_xy(U.m, xx, yy);
            float rx = w.x - c.x, ry = w.y - c.y;
            float torque = rx * fy - ry * fx;
            if (id >= 0 && id < EFL_MAX_SOLIDS) {
                atomicAdd(&sb[id], f2i(fx * 10.0f));
                atomicAdd(&sb[EFL_MAX_SOLIDS + id], f2i(fy * 10.0f));
                atomicAdd(&sb[2 * EFL_MAX_SOLIDS + id], f2i(torque * 10.0f));
                touched = 1;
            }
        }
    }
    __syncthreads();
    if (!touched) return;
    for (int i = tid; i < 3 * EFL_MAX_SOLIDS; i += nth)
        if (sb[i] != 0) atomicAdd(&bins[i], sb[i]);
}
// accumulate_forces.wgsl:16-32
__global__ void k_accumulate_forces(const int* bins, efl_solid_force* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= EFL_MAX_SOLIDS) return;
    efl_solid_force f;
    f.force[0] = (float)bins[i] * 0.1f;
    f.force[1] = (float)bins[EFL_MAX_SOLIDS + i] * 0.1f;
    f.torque = (float)bins[2 * EFL_MAX_SOLIDS + i] * 0.1f;
    f._pad = 0.0f;
    out[i] = f;
}

// calculate_volume.wgsl:11-75 as an exact integer count of phi < 0.
__global__ void k_volume(PF ls0, unsigned long long* out) {
    int x = gx(), y = gy();
    unsigned long long c = (x < ls0.w && y < ls0.h && ls0.at(x, y) < 0.0f) ? 1ull : 0ull;
    unsigned mask = __ballot_sync(0xffffffffu, c != 0);
    if ((threadIdx.x & 31) == 0 && mask) atomicAdd(out, (unsigned long long)__popc(mask));
}

// diagnostics/{min,max}_velocity.wgsl partial_reduction: one 16 x 16 block
// per workgroup; min over fluid cells (1e30 elsewhere), max over all cells.
__global__ void __launch_bounds__(256) k_velocity_partial(PF u, PF v, PF ls, float* pmin, float* pmax) {
    __shared__ float smin[256], smax[256];
    const int x = blockIdx.x * 16 + threadIdx.x, y = blockIdx.y * 16 + threadIdx.y;
    const int lid = threadIdx.y * 16 + threadIdx.x;
    const float u0 = 0.5f * (u.ld(x, y) + u.ld(x + 1, y));
    const float v0 = 0.5f * (v.ld(x, y) + v.ld(x, y + 1));
    const float mag = sqrtf(u0 * u0 + v0 * v0);
    smin[lid] = ls.ld(x, y) < 0.0f ? mag : 1e30f;
    smax[lid] = mag;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (lid < st) {
            smin[lid] = fminf(smin[lid], smin[lid + st]);
            smax[lid] = fmaxf(smax[lid], smax[lid + st]);
        }
        __syncthreads();
    }
    if (lid == 0) {
        const int w = blockIdx.x + blockIdx.y * gridDim.x;
        pmin[w] = smin[0];
        pmax[w] = smax[0];
    }
}
// diagnostics/{min,max}_velocity.wgsl reduction: 512 lanes each ADD their
// partials i = lane, lane + 512, ... from 0.0 (as the reference does), then min / max.
__global__ void __launch_bounds__(512) k_velocity_final(const float* pmin, const float* pmax, int n, float* out) {
    __shared__ float smin[512], smax[512];
    const int lid = threadIdx.x;
    float a = 0.0f, b = 0.0f;
    for (int i = lid; i < n; i += 512) {
        a += pmin[i];
        b += pmax[i];
    }
    smin[lid] = a;
    smax[lid] = b;
    __syncthreads();
    for (int st = 256; st > 0; st >>= 1) {
        if (lid < st) {
            smin[lid] = fminf(smin[lid], smin[lid + st]);
            smax[lid] = fmaxf(smax[lid], smax[lid + st]);
        }
        __syncthreads();
    }
    if (lid == 0) {
        out[0] = smin[0];
        out[1] = smax[0];
    }
}

}  // namespace efl
