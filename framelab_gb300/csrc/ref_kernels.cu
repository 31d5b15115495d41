// ref_kernels.cu -- GPU kernels that reproduce the reference's CPU projectors
// bit for bit (FL_MODEL_SIDDON_REF forward, FL_MODEL_CHORD_REF adjoint).
//
// Every float operation is the one the reference performs, in its order,
// through the pinned intrinsics of fl_common.cuh (no FMA contraction).
// Work that cannot change the result is skipped: the Siddon merge starts a
// few planes before the ray enters the image and stops a few planes after it
// leaves (decided in FP64 with a 2-voxel safety band), since segments
// outside the image add nothing in the reference either.
#include "fl_common.cuh"
#include "fl_plan.h"

namespace {

// ---------------------------------------------------------------------------
// Siddon merge (version 0). One axis of plane crossings; see oracle.c for the
// argument that a plain sorted merge equals the reference's sort_alpha() merge
// (sort_alpha.cpp:15-60) for the sum it feeds.
// ---------------------------------------------------------------------------
struct MergeAxis {
    int i;        // current plane index
    int left;     // planes still to emit (including i)
    int di;       // +1 / -1
    float p1, d;  // source coordinate, direction component
    float pitch;  // plane spacing: 1 for x/y, dz0 for z
    bool zaxis;
    float head;
};

__device__ __forceinline__ float merge_alpha(const MergeAxis& a, int i)
{
    if (a.zaxis) return fdiv(fsub(fmul((float)i, a.pitch), a.p1), a.d);  // Ax_cone_mf_cpu_siddon.cpp:69
    return fdiv(fsub((float)i, a.p1), a.d);                               // Ax_fan_mf_cpu_siddon.cpp:44
}

// Box-clip one axis of the ray (p1 -> p1+d) against planes [lo, hi] in FP64;
// returns false when the ray misses the slab entirely.
__device__ __forceinline__ bool clip_axis(double p1, double d, double lo, double hi,
                                          double& amin, double& amax)
{
    if (d == 0.0) return p1 >= lo && p1 <= hi;
    double t0 = (lo - p1) / d, t1 = (hi - p1) / d;
    if (t0 > t1) { double t = t0; t0 = t1; t1 = t; }
    amin = fmax(amin, t0);
    amax = fmin(amax, t1);
    return true;
}

// Plane index range [first..last] (in traversal order) covering alpha in
// [A0, A1] plus one plane on either side and one more for rounding.
__device__ __forceinline__ void init_axis(MergeAxis& a, float p1, float p2, int n, bool zaxis,
                                          float dz0, double A0, double A1)
{
    int n2 = n / 2;
    a.p1 = p1; a.d = fsub(p2, p1); a.zaxis = zaxis; a.pitch = zaxis ? dz0 : 1.0f;
    a.left = 0;
    if (p1 == p2) return;
    double pitch = zaxis ? (double)dz0 : 1.0;
    double c0 = ((double)p1 + A0 * (double)a.d) / pitch;
    double c1 = ((double)p1 + A1 * (double)a.d) / pitch;
    int first, last;
    if (p1 < p2) {
        a.di = 1;
        first = max(-n2, (int)floor(c0) - 2);
        last = min(n2, (int)ceil(c1) + 2);
        a.left = last - first + 1;
    } else {
        a.di = -1;
        first = min(n2, (int)ceil(c0) + 2);
        last = max(-n2, (int)floor(c1) - 2);
        a.left = first - last + 1;
    }
    if (a.left < 0) a.left = 0;
    a.i = first;
    if (a.left > 0) a.head = merge_alpha(a, a.i);
}

template <int NA>
__device__ __forceinline__ int pick_min(const MergeAxis (&ax)[NA])
{
    int best = -1;
#pragma unroll
    for (int k = 0; k < NA; k++)
        if (ax[k].left > 0 && (best < 0 || ax[k].head < ax[best].head)) best = k;
    return best;
}

template <int NA>
__device__ __forceinline__ float pop(MergeAxis (&ax)[NA], int k)
{
    float v = ax[k].head;
    // select by constant index so the array stays in registers
#pragma unroll
    for (int j = 0; j < NA; j++) {
        if (j == k) {
            ax[j].left -= 1;
            ax[j].i += ax[j].di;
            if (ax[j].left > 0) ax[j].head = merge_alpha(ax[j], ax[j].i);
        }
    }
    return v;
}

// Fan-beam Siddon, restating Ax_fan_mf_cpu_siddon.cpp:19-93. One thread per ray.
__global__ void __launch_bounds__(128)
k_ref_fan_siddon(const float* __restrict__ X, float* __restrict__ y,
                 const float* __restrict__ cphi_v, const float* __restrict__ sphi_v,
                 const float* __restrict__ ydet, const int* __restrict__ vframe, float SO,
                 float OD, float scale, int nx, int ny, int nd, long long nper)
{
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    int iv = blockIdx.y;
    if (id >= nd) return;
    const float* x = X + (long long)vframe[iv] * nper;
    float c = cphi_v[iv], s = sphi_v[iv];
    float x1 = fmul(c, -SO), y1 = fmul(s, -SO);
    float u = ydet[id];
    float x2 = fsub(fmul(c, OD), fmul(s, u));
    float y2 = fadd(fmul(s, OD), fmul(c, u));
    float dx = fsub(x2, x1), dy = fsub(y2, y1);
    float total = fsqrt(fadd(fmul(dx, dx), fmul(dy, dy)));
    int nx2 = nx / 2, ny2 = ny / 2;

    double A0 = -1e300, A1 = 1e300;
    bool hit = clip_axis(x1, dx, -nx2 - 2.0, nx - nx2 + 2.0, A0, A1) &&
               clip_axis(y1, dy, -ny2 - 2.0, ny - ny2 + 2.0, A0, A1);
    float acc = 0.0f;
    if (hit && A0 < A1) {
        MergeAxis ax[2];
        init_axis(ax[0], x1, x2, nx, false, 1.0f, A0, A1);
        init_axis(ax[1], y1, y2, ny, false, 1.0f, A0, A1);
        int k = pick_min(ax);
        if (k >= 0) {
            float prev = pop(ax, k);
            while ((k = pick_min(ax)) >= 0) {
                float next = pop(ax, k);
                float ac = fmul(0.5f, fadd(prev, next));
                int tx = (int)floorf(fadd(fadd(x1, fmul(ac, dx)), (float)nx2));
                if (tx >= 0 && tx < nx) {
                    int ty = (int)floorf(fadd(fadd(y1, fmul(ac, dy)), (float)ny2));
                    if (ty >= 0 && ty < ny) {
                        float seg = fmul(fsub(next, prev), total);
                        acc = fadd(acc, fmul(seg, __ldg(x + ty * nx + tx)));
                    }
                }
                prev = next;
            }
        }
    }
    y[(long long)iv * nd + id] = fmul(acc, scale);
}

// Cone-beam Siddon, restating Ax_cone_mf_cpu_siddon.cpp:19-134.
__global__ void __launch_bounds__(128)
k_ref_cone_siddon(const float* __restrict__ X, float* __restrict__ y,
                  const float* __restrict__ cphi_v, const float* __restrict__ sphi_v,
                  const float* __restrict__ sdz, const float* __restrict__ ydet,
                  const float* __restrict__ zdet, const int* __restrict__ vframe, float SO,
                  float OD, float scale, int nx, int ny, int nz, float dz0, int na, int nb,
                  long long nper)
{
    int ia = blockIdx.x * blockDim.x + threadIdx.x;
    int ib = blockIdx.y;
    int iv = blockIdx.z;
    if (ia >= na) return;
    const float* x = X + (long long)vframe[iv] * nper;
    float c = cphi_v[iv], s = sphi_v[iv];
    float x1 = fmul(c, -SO), y1 = fmul(s, -SO), z1 = sdz[iv];
    float u = ydet[ia];
    float x2 = fsub(fmul(c, OD), fmul(s, u));
    float y2 = fadd(fmul(s, OD), fmul(c, u));
    float z2 = fadd(zdet[ib], sdz[iv]);
    float dx = fsub(x2, x1), dy = fsub(y2, y1), dz = fsub(z2, z1);
    float total = fsqrt(fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fmul(dz, dz)));
    int nx2 = nx / 2, ny2 = ny / 2, nz2 = nz / 2;

    double A0 = -1e300, A1 = 1e300;
    bool hit = clip_axis(x1, dx, -nx2 - 2.0, nx - nx2 + 2.0, A0, A1) &&
               clip_axis(y1, dy, -ny2 - 2.0, ny - ny2 + 2.0, A0, A1) &&
               clip_axis(z1, dz, (-nz2 - 2.0) * (double)dz0, (nz - nz2 + 2.0) * (double)dz0,
                         A0, A1);
    float acc = 0.0f;
    if (hit && A0 < A1) {
        MergeAxis ax[3];
        init_axis(ax[0], x1, x2, nx, false, 1.0f, A0, A1);
        init_axis(ax[1], y1, y2, ny, false, 1.0f, A0, A1);
        init_axis(ax[2], z1, z2, nz, true, dz0, A0, A1);
        int k = pick_min(ax);
        if (k >= 0) {
            float prev = pop(ax, k);
            while ((k = pick_min(ax)) >= 0) {
                float next = pop(ax, k);
                float ac = fmul(0.5f, fadd(prev, next));
                int tx = (int)floorf(fadd(fadd(x1, fmul(ac, dx)), (float)nx2));
                if (tx >= 0 && tx < nx) {
                    int ty = (int)floorf(fadd(fadd(y1, fmul(ac, dy)), (float)ny2));
                    if (ty >= 0 && ty < ny) {
                        int tz = (int)floorf(fadd(fdiv(fadd(z1, fmul(ac, dz)), dz0), (float)nz2));
                        if (tz >= 0 && tz < nz) {
                            float seg = fmul(fsub(next, prev), total);
                            acc = fadd(acc, fmul(seg, __ldg(x + ((long long)tz * ny + ty) * nx + tx)));
                        }
                    }
                }
                prev = next;
            }
        }
    }
    y[((long long)iv * nb + ib) * na + ia] = fmul(acc, scale);
}

// ---------------------------------------------------------------------------
// Chord-length backprojectors (version 1).
// ---------------------------------------------------------------------------

// find_l (find_l.cpp:18-45): chord of the line a*x+b*y=c through the unit
// pixel centred at (x, y).
__device__ __forceinline__ float chord_unit_pixel(float a, float b, float c, float x, float y)
{
    float aa = fabs_ref(a), bb = fabs_ref(b);
    float ha = fdiv(aa, 2.0f), hb = fdiv(bb, 2.0f);
    float reach = fadd(ha, hb);
    float d = fabs_ref(fsub(fsub(c, fmul(a, x)), fmul(b, y)));
    if (!(d < reach)) return 0.0f;
    float flat = fabs_ref(fsub(ha, hb));
    float full = (ha < hb) ? fdiv(1.0f, bb) : fdiv(1.0f, aa);
    return (d <= flat) ? full : fdiv(fsub(reach, d), fmul(aa, bb));
}

// 2-D helper of find_l_3d.cpp:19-92 (a line through a w x h rectangle).
__device__ float chord_rect(float px, float py, float qx, float qy, float w, float h, float x,
                            float y)
{
    float a = fsub(qx, px), b = fsub(qy, py);
    float hw = fdiv(w, 2.0f), hh = fdiv(h, 2.0f);
    if (a == 0.0f) return (fabs_ref(fsub(px, x)) <= hw) ? h : 0.0f;
    if (b == 0.0f) return (fabs_ref(fsub(py, y)) <= hh) ? w : 0.0f;
    float rx = fsub(px, x), ry = fsub(py, y);
    float hx0 = 0, hy0 = 0, hx1 = 0, hy1 = 0;
    int nh = 0;
    bool xfirst = fabs_ref(a) > fabs_ref(b);
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
        if (pass == 1 && nh >= 2) break;
        bool xfam = (pass == 0) ? xfirst : !xfirst;
        float s, t, uu;
        if (xfam) { s = fdiv(b, a); t = fadd(fmul(s, -rx), ry); uu = fmul(s, hw); }
        else      { s = fdiv(a, b); t = fadd(fmul(s, -ry), rx); uu = fmul(s, hh); }
#pragma unroll
        for (int side = 0; side < 2; side++) {
            if (pass == 1 && side == 1 && nh >= 2) break;
            float v = side ? fadd(t, uu) : fsub(t, uu);
            bool ok = xfam ? (fabs_ref(v) <= hh) : (fabs_ref(v) <= hw);
            if (ok) {
                float px_ = xfam ? (side ? hw : -hw) : v;
                float py_ = xfam ? v : (side ? hh : -hh);
                if (nh == 0) { hx0 = px_; hy0 = py_; } else { hx1 = px_; hy1 = py_; }
                nh++;
            }
        }
    }
    if (nh != 2) return 0.0f;
    float ex = fsub(hx1, hx0), ey = fsub(hy1, hy0);
    return fsqrt(fadd(fmul(ex, ex), fmul(ey, ey)));
}

// find_l_3d (find_l_3d.cpp:94-182): chord of the line P->Q through the box of
// size (w,h,t) centred at (x,y,z); faces of the dominant xy axis first, then
// the other xy axis, then z; the first two hits give the chord.
__device__ float chord_box(float px, float py, float pz, float qx, float qy, float qz, float w,
                           float h, float t, float x, float y, float z)
{
    float a = fsub(qx, px), b = fsub(qy, py), c = fsub(qz, pz);
    float hw = fdiv(w, 2.0f), hh = fdiv(h, 2.0f), ht = fdiv(t, 2.0f);
    if (a == 0.0f) return chord_rect(py, pz, qy, qz, h, t, y, z);
    if (b == 0.0f) return chord_rect(px, pz, qx, qz, w, t, x, z);
    float rx = fsub(px, x), ry = fsub(py, y), rz = fsub(pz, z);
    float P0[3] = {0, 0, 0}, P1[3] = {0, 0, 0};
    int nh = 0;
    int f0 = (fabs_ref(a) > fabs_ref(b)) ? 0 : 1;
#pragma unroll
    for (int pass = 0; pass < 3; pass++) {
        if (pass > 0 && nh >= 2) break;
        int fam = (pass == 0) ? f0 : (pass == 1 ? 1 - f0 : 2);
        float u0, u1, v0, v1, lim0, lim1;
        if (fam == 0) {
            float s = fdiv(b, a); u0 = fadd(fmul(s, -rx), ry); u1 = fmul(s, hw);
            s = fdiv(c, a);       v0 = fadd(fmul(s, -rx), rz); v1 = fmul(s, hw);
            lim0 = hh; lim1 = ht;
        } else if (fam == 1) {
            float s = fdiv(a, b); u0 = fadd(fmul(s, -ry), rx); u1 = fmul(s, hh);
            s = fdiv(c, b);       v0 = fadd(fmul(s, -ry), rz); v1 = fmul(s, hh);
            lim0 = hw; lim1 = ht;
        } else {
            float s = fdiv(a, c); u0 = fadd(fmul(s, -rz), rx); u1 = fmul(s, ht);
            s = fdiv(b, c);       v0 = fadd(fmul(s, -rz), ry); v1 = fmul(s, ht);
            lim0 = hw; lim1 = hh;
        }
#pragma unroll
        for (int side = 0; side < 2; side++) {
            if (pass > 0 && side == 1 && nh >= 2) break;
            float uu = side ? fadd(u0, u1) : fsub(u0, u1);
            float vv = side ? fadd(v0, v1) : fsub(v0, v1);
            if (fabs_ref(uu) <= lim0 && fabs_ref(vv) <= lim1) {
                float q0, q1, q2;
                if (fam == 0)      { q0 = side ? hw : -hw; q1 = uu; q2 = vv; }
                else if (fam == 1) { q0 = uu; q1 = side ? hh : -hh; q2 = vv; }
                else               { q0 = uu; q1 = vv; q2 = side ? ht : -ht; }
                if (nh == 0) { P0[0] = q0; P0[1] = q1; P0[2] = q2; }
                else         { P1[0] = q0; P1[1] = q1; P1[2] = q2; }
                nh++;
            }
        }
    }
    if (nh != 2) return 0.0f;
    float ex = fsub(P1[0], P0[0]), ey = fsub(P1[1], P0[1]), ez = fsub(P1[2], P0[2]);
    return fsqrt(fadd(fadd(fmul(ex, ex), fmul(ey, ey)), fmul(ez, ez)));
}

// One detector column of a voxel column's window in one view: what find_l_3d
// (w = h = t = 1) needs of it, and where its rays pass (k_ref_cone_chord_adj).
struct alignas(16) ChordCol {
    float a, b;                    // direction
    float t0, k, half;             // parameter nearest the voxel column, reach, 1/2 + margin
    float cmin, cmax;              // row directions c for which the reach holds
    int ia, flags, pad;
    union {
        struct {                   // any column
            float uxm, uxp, uym, uyp;   // crossings at the faces x = -+1/2 (y) and y = -+1/2 (x)
            float x2, y2;               // detector point
        };
        struct {                   // kTwo: the two faces the rays pass, in the order tested
            float d1, i1, o1, h1;       // direction component, its reciprocal, source offset, -+1/2
            float d2, i2, o2, h2;
            float p1x, p1y, p2x, p2y;   // where the rays pass them
            float e2;                   // (p2x - p1x)^2 + (p2y - p1y)^2
        };
    };
};
enum { kXm = 1, kXp = 2, kYm = 4, kYp = 8,    // the crossing lies within the face's width
       kXFirst = 16,                          // |a| > |b|: the x faces are tested first
       kAxis = 32,                            // a = 0 or b = 0: find_l_3d's 2-D cases
       kRowsSafe = 64,                        // every row's direction is in [cmin, cmax] or 0
       kTwo = 128 };                          // chord_two applies to every row

// n / d, correctly rounded, from the correctly rounded reciprocal i of d: with q
// = RN(n i) within an ulp of n / d and the remainder n - q d exact, RN(q + (n -
// q d) i) is RN(n / d) (P. Markstein, IBM J. Res. Dev. 34, 1990, theorem 8). Both
// operands and the quotient are far from the ends of the exponent range here
// (kRowsSafe); n = 0 gives 0.
__device__ __forceinline__ float div_by(float n, float d, float i)
{
    const float q = fmul(n, i);
    return __fmaf_rn(__fmaf_rn(-q, d, n), i, q);
}

// find_l_3d for a column whose rays pass exactly two faces in the plane, with
// |c| below |a| or |b| / 1.2 in every row: the two faces' hits, or one of them
// and a z face's (two z hits alone are a run (a / c, b / c) of more than one
// voxel: none, or a third hit: no chord). The same float expressions as
// chord_box, in its order.
__device__ __forceinline__ float chord_two(const ChordCol& q, float c, float rx, float ry, float rz)
{
    const float s1 = div_by(c, q.d1, q.i1), s2 = div_by(c, q.d2, q.i2);
    const float v1 = fadd(fadd(fmul(s1, -q.o1), rz), fmul(s1, q.h1));
    const float v2 = fadd(fadd(fmul(s2, -q.o2), rz), fmul(s2, q.h2));
    const bool k1 = fabs_ref(v1) <= 0.5f, k2 = fabs_ref(v2) <= 0.5f;
    if (k1 && k2) {
        const float ez = fsub(v2, v1);
        return fsqrt(fadd(q.e2, fmul(ez, ez)));
    }
    if (!k1 && !k2) return 0.0f;
    const float px = k1 ? q.p1x : q.p2x, py = k1 ? q.p1y : q.p2y, pz = k1 ? v1 : v2;
    const float ic = fdiv(1.0f, c);
    const float su = div_by(q.a, c, ic), sv = div_by(q.b, c, ic);
    const float u0 = fadd(fmul(su, -rz), rx), u1 = fmul(su, 0.5f);
    const float v0 = fadd(fmul(sv, -rz), ry), w1 = fmul(sv, 0.5f);
    const float um = fsub(u0, u1), vm = fsub(v0, w1), up = fadd(u0, u1), vp = fadd(v0, w1);
    const bool lo = fabs_ref(um) <= 0.5f && fabs_ref(vm) <= 0.5f;
    const bool hi = fabs_ref(up) <= 0.5f && fabs_ref(vp) <= 0.5f;
    if (!lo && !hi) return 0.0f;
    const float ex = fsub(lo ? um : up, px), ey = fsub(lo ? vm : vp, py);
    const float ez = fsub(lo ? -0.5f : 0.5f, pz);
    return fsqrt(fadd(fadd(fmul(ex, ex), fmul(ey, ey)), fmul(ez, ez)));
}

// chord_box for a unit cube when the in-plane direction (a, b) has no zero
// component: every value is the same float expression chord_box evaluates, in
// its order of faces, so the result has the same bits. The in-plane crossings
// and whether they pass come with the column; a family whose two crossings both
// fail has no hit and needs no division. Two hits on the z faces alone are a
// chord whose in-plane run (a / c, b / c) is at most one voxel in x and y, so
// without a hit before them the z faces are only tested where |c| can be as
// large as |a| and |b| (one hit gives no chord).
__device__ __forceinline__ float chord_box_col(const ChordCol& q, float c, float rx, float ry,
                                               float rz)
{
    float P0[3] = {0, 0, 0}, P1[3] = {0, 0, 0};
    int nh = 0;
    auto hit = [&](float x, float y, float z) {
        if (nh == 0) { P0[0] = x; P0[1] = y; P0[2] = z; }
        else         { P1[0] = x; P1[1] = y; P1[2] = z; }
        nh++;
    };
    const int f = q.flags;
    auto xfaces = [&](bool all) {
        if (!(f & (kXm | kXp))) return;
        const float s = fdiv(c, q.a), v0 = fadd(fmul(s, -rx), rz), v1 = fmul(s, 0.5f);
        const float vm = fsub(v0, v1), vp = fadd(v0, v1);
        if ((f & kXm) && fabs_ref(vm) <= 0.5f) hit(-0.5f, q.uxm, vm);
        if ((all || nh < 2) && (f & kXp) && fabs_ref(vp) <= 0.5f) hit(0.5f, q.uxp, vp);
    };
    auto yfaces = [&](bool all) {
        if (!(f & (kYm | kYp))) return;
        const float s = fdiv(c, q.b), v0 = fadd(fmul(s, -ry), rz), v1 = fmul(s, 0.5f);
        const float vm = fsub(v0, v1), vp = fadd(v0, v1);
        if ((f & kYm) && fabs_ref(vm) <= 0.5f) hit(q.uym, -0.5f, vm);
        if ((all || nh < 2) && (f & kYp) && fabs_ref(vp) <= 0.5f) hit(q.uyp, 0.5f, vp);
    };
    if (f & kXFirst) { xfaces(true); if (nh < 2) yfaces(false); }
    else             { yfaces(true); if (nh < 2) xfaces(false); }
    if (nh == 0 && fmaxf(fabsf(q.a), fabsf(q.b)) > 1.2f * fabsf(c)) return 0.0f;
    if (nh < 2) {
        float s = fdiv(q.a, c);
        const float u0 = fadd(fmul(s, -rz), rx), u1 = fmul(s, 0.5f);
        s = fdiv(q.b, c);
        const float v0 = fadd(fmul(s, -rz), ry), v1 = fmul(s, 0.5f);
        const float um = fsub(u0, u1), up = fadd(u0, u1), vm = fsub(v0, v1), vp = fadd(v0, v1);
        if (fabs_ref(um) <= 0.5f && fabs_ref(vm) <= 0.5f) hit(um, vm, -0.5f);
        if (nh < 2 && fabs_ref(up) <= 0.5f && fabs_ref(vp) <= 0.5f) hit(up, vp, 0.5f);
    }
    if (nh != 2) return 0.0f;
    const float ex = fsub(P1[0], P0[0]), ey = fsub(P1[1], P0[1]), ez = fsub(P1[2], P0[2]);
    return fsqrt(fadd(fadd(fmul(ex, ex), fmul(ey, ey)), fmul(ez, ez)));
}

// Fan-beam chord backprojection, restating Atx_fan_mf_cpu_new.cpp:21-63.
// One thread per (pixel, frame).
__global__ void __launch_bounds__(128)
k_ref_fan_chord_adj(float* __restrict__ x, const float* __restrict__ Y,
                    const float* __restrict__ cos_phi, const float* __restrict__ sin_phi,
                    const float* __restrict__ cos_det, const float* __restrict__ sin_det,
                    const int* __restrict__ idY, const int* __restrict__ Nv, int tmp_size,
                    float SO, float OD, float scale, float dy_det, float y_os, int nx, int ny,
                    int nd, int nt)
{
    int ix = blockIdx.x * blockDim.x + threadIdx.x;
    int iy = blockIdx.y;
    int it = blockIdx.z;
    if (ix >= nx) return;
    int nd2 = nd / 2, nx2 = nx / 2, ny2 = ny / 2;
    float SD = fadd(SO, OD);
    // (float)(i + 0.5 - n2) is exact for any realistic size
    float yc = (float)(iy - ny2) + 0.5f;
    float xc = (float)(ix - nx2) + 0.5f;
    float acc = 0.0f;
    int nvf = Nv[it];
    for (int j = 0; j < nvf; j++) {
        int iv = idY[it * tmp_size + j];
        const float* yv = Y + (long long)iv * nd;
        float c = cos_phi[iv], s = sin_phi[iv];
        float xr = fadd(fmul(c, xc), fmul(s, yc));
        float yr = fadd(fmul(-s, xc), fmul(c, yc));
        float g = fdiv(SD, fmul(fadd(xr, SO), dy_det));
        int hi = (int)floorf(fadd(fsub(fmul(fadd(yr, 1.0f), g), y_os), (float)nd2));
        int lo = (int)floorf(fadd(fsub(fmul(fsub(yr, 1.0f), g), y_os), (float)nd2));
        lo = max(lo, 0);
        hi = min(hi, nd - 1);
        for (int id = lo; id <= hi; id++) {
            float sd = __ldg(sin_det + id), cd = __ldg(cos_det + id);
            float Px = -fadd(fmul(sd, c), fmul(cd, s));
            float Py = fsub(fmul(cd, c), fmul(sd, s));
            float Pd = fmul(SO, sd);
            float l = chord_unit_pixel(Px, Py, Pd, xc, yc);
            if (l > 0.0f) acc = fadd(acc, fmul(l, __ldg(yv + id)));
        }
    }
    x[(long long)it * nx * ny + (long long)iy * nx + ix] = fmul(acc, scale);
}

// Prepares a cone sinogram for the backprojection below: whether every value is
// finite (flag[0 .. nflag), all 0 before, becomes 1 when one is not), and with RF the
// rows-fastest copy yt[(iv na + ia) nb + ib] = y[(iv nb + ib) na + ia], 32 x 32 tiles
// through shared memory. Without scratch the flag is the backprojection's own
// output, every voxel of it, read by its voxel's lane before it is written. Blocks
// that find such a value write the same flags; one that sees that another has begun
// leaves it to that one.
template <bool RF, typename F>
__global__ void __launch_bounds__(256)
k_ref_prepare(const float* __restrict__ y, float* __restrict__ yt, int na, int nb, F* flag,
              long long nflag)
{
    __shared__ float tile[RF ? 32 : 1][33];
    const int a0 = blockIdx.x * 32, b0 = blockIdx.y * 32;
    const long long base = (long long)blockIdx.z * na * nb;
    bool fin = true;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int ia = a0 + threadIdx.x, ib = b0 + k;
        if (ia >= na || ib >= nb) continue;
        const float v = y[base + (long long)ib * na + ia];
        if (RF) tile[k][threadIdx.x] = v;
        fin = fin && isfinite(v);
    }
    const bool all = __syncthreads_and(fin);
    if (RF)
        for (int k = threadIdx.y; k < 32; k += 8) {
            const int ia = a0 + k, ib = b0 + threadIdx.x;
            if (ia < na && ib < nb) yt[base + (long long)ia * nb + ib] = tile[threadIdx.x][k];
        }
    if (all || __syncthreads_or(*(volatile F*)flag != F(0))) return;    // (all or none of the block)
    for (long long k = threadIdx.y * 32 + threadIdx.x; k < nflag; k += 256) flag[k] = F(1);
}

constexpr int kChordWarps = 4;     // neighbouring voxel columns per thread block

// Cone-beam chord backprojection, restating Atx_cone_mf_cpu_new.cpp:23-85
// (unit-cube chord, z window half-width sqrt(1 + dz^2/2)). A warp takes one
// voxel column, a lane one voxel (groups of 2^lz lanes where the volume is
// low): the detector columns of a view's window and their row-independent
// find_l_3d terms are the same for all its voxels, so the lanes compute them
// once, one column each, for several views together. The sums run in the
// reference's order: rows, then columns.
//
// Rays that miss the voxel are not evaluated. The reference's window is about
// 5 x 6 rays per voxel and view at a magnification of two, of which about 5
// meet it; the others get l = 0 from find_l_3d and add an exact zero (unless a
// value is not finite: k_ref_prepare turns the skipping off). A line that misses the
// voxel's box grown by a margin m on every side passes none of the reference's
// face tests: a test computes u = s (h - r) + r' for a slope s of the direction
// (a, b, c) and offsets r, r' of the source, with an error of at most 2^-22
// (|s| (|r| + 1/2) + |r'|); where the test could pass, |u| <= 1/2, so |s r| <=
// |r'| + |s| / 2 + 1. With slopes and offsets below L that is 2^-22 (3 L / 2 +
// 1) and the comparisons below carry less than 2^-21 L themselves: under 0.02
// for L = 1e4 and 0.12 for L = 1e5, the two margins used. Rays with a larger
// slope (a row at c = 0 exactly fails the z faces by inf or NaN) take the full
// test.
//   in xy: |a ry - b rx| > (|a| + |b|) (1/2 + m);
//   in z:  every point of the line inside the grown square lies within 0.88 of
//          the one nearest its centre, at t0: |rz + c t0| > 1/2 + m + |c| k,
//          k = 0.88 / |(a, b)|.
// zmin, zmax: the smallest non-zero and the largest |z_det|. RF: Y has its
// rows fastest and *bad is the flag, else its columns (k_ref_prepare).
// Bound: issue (82-85 %; 871 warp instructions per column of 32 voxels and
// view). 128^3, 120 views, 192 x 160 panel: 27.6 ms with a thread per voxel,
// the window's columns set up by each and every ray of it evaluated; 14.2 with
// this mapping and the skipping ray by ray; 10.1 with the rows narrowed first
// and no division for faces that fail in the plane; 8.30 with chord_two; 6.43
// with the margin of 0.02 and without the per-ray test where chord_two applies.
// 6 and 10 blocks per SM 6.68 and 6.61. 200^3, 40 views, 400 x 300: 51.8 -> 10.6.
template <bool RF>
__global__ void __launch_bounds__(kChordWarps * 32, 8)
k_ref_cone_chord_adj(float* __restrict__ x, const float* __restrict__ Y,
                     const int* __restrict__ bad, const float* __restrict__ cos_phi,
                     const float* __restrict__ sin_phi, const float* __restrict__ sdz,
                     const float* __restrict__ ydet, const float* __restrict__ zdet,
                     const int* __restrict__ idY, const int* __restrict__ Nv, int tmp_size,
                     float SO, float OD, float scale, float dy_det, float y_os, float dz_det,
                     float dz, int nx, int ny, int nz, int na, int nb, float zmin, float zmax,
                     int rows_uniform, float dv0, float inv_dv, int zruns, int lz)
{
    __shared__ ChordCol cols[kChordWarps][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int ZL = 1 << lz, g0 = lane & ~(ZL - 1), sub = lane & (ZL - 1);
    const unsigned gm = (0xffffffffu >> (32 - ZL)) << g0;
    const int ix = ((blockIdx.x * kChordWarps + wp) << (5 - lz)) + (g0 >> lz);
    const int iy = blockIdx.y;
    const int iz = ((int)(blockIdx.z % zruns) << lz) + sub, it = blockIdx.z / zruns;
    if (ix >= nx) return;                               // whole groups
    const bool on = iz < nz;
    const bool skip = RF ? !*bad
                         : x[(long long)it * nx * ny * nz + ((long long)min(iz, nz - 1) * ny + iy) * nx + ix] == 0.0f;
    if (!RF) __syncwarp(gm);                            // read before any lane stores its sum
    const float SD = fadd(SO, OD);
    const int na2 = na / 2, nb2 = nb / 2, nx2 = nx / 2, ny2 = ny / 2, nz2 = nz / 2;
    const long long nd = (long long)na * nb;
    const float dwin = fsqrt(fadd(1.0f, fdiv(fmul(dz, dz), 2.0f)));
    const float zc = fmul((float)(iz - nz2) + 0.5f, dz);
    const float yc = (float)(iy - ny2) + 0.5f, xc = (float)(ix - nx2) + 0.5f;
    float acc = 0.0f;
    const int nvf = Nv[it];
    for (int jb = 0; jb < nvf; jb += ZL) {
        // this lane's view and its window of detector columns
        int iv = 0, amin = 0, amax = -1;
        if (jb + sub < nvf) {
            iv = idY[it * tmp_size + jb + sub];
            const float c = cos_phi[iv], s = sin_phi[iv];
            const float xr = fadd(fmul(c, xc), fmul(s, yc));
            const float yr = fadd(fmul(-s, xc), fmul(c, yc));
            const float g = fdiv(SD, fmul(fadd(xr, SO), dy_det));
            amax = (int)floorf(fadd(fsub(fmul(fadd(yr, 1.0f), g), y_os), (float)na2));
            amin = (int)floorf(fadd(fsub(fmul(fsub(yr, 1.0f), g), y_os), (float)na2));
            // into [0, na] and [-1, na - 1]: both ends can be as large as an int holds
            // (a very fine panel, a source inside the volume), and lanes are added
            amin = min(max(amin, 0), na); amax = max(min(amax, na - 1), -1);
        }
        const int maxw = __reduce_max_sync(gm, amax - amin + 1);
        if (maxw <= 0) continue;
        int lg = 2;                                     // 4 .. ZL columns per view
        while (lg < lz && (1 << lg) < maxw) lg++;
        const int W = 1 << lg;
        for (int v0 = 0; v0 < min(ZL, nvf - jb); v0 += ZL >> lg) {
            const int vm = g0 + v0 + (sub >> lg);
            const int lo = __shfl_sync(gm, amin, vm), hi = __shfl_sync(gm, amax, vm);
            const int ivm = __shfl_sync(gm, iv, vm);
            const int ia = lo + (sub & (W - 1));
            bool ok = ia <= hi;
            __syncwarp(gm);
            if (ok) {
                const float c = cos_phi[ivm], s = sin_phi[ivm];
                const float x1 = fmul(c, -SO), y1 = fmul(s, -SO), z1 = sdz[ivm];
                const float rx = fsub(x1, xc), ry = fsub(y1, yc);
                const float u = __ldg(ydet + ia);
                ChordCol q;
                q.x2 = fsub(fmul(c, OD), fmul(s, u)); q.y2 = fadd(fmul(s, OD), fmul(c, u));
                q.a = fsub(q.x2, x1); q.b = fsub(q.y2, y1);
                const float aa = fabsf(q.a), bb = fabsf(q.b);
                q.flags = (q.a == 0.0f || q.b == 0.0f) ? kAxis : aa > bb ? kXFirst : 0;
                q.uxm = q.uxp = q.uym = q.uyp = 0.0f;
                if (!(q.flags & kAxis)) {
                    float w = fdiv(q.b, q.a);
                    float u0 = fadd(fmul(w, -rx), ry), u1 = fmul(w, 0.5f);
                    q.uxm = fsub(u0, u1); q.uxp = fadd(u0, u1);
                    w = fdiv(q.a, q.b);
                    u0 = fadd(fmul(w, -ry), rx); u1 = fmul(w, 0.5f);
                    q.uym = fsub(u0, u1); q.uyp = fadd(u0, u1);
                    q.flags |= (fabsf(q.uxm) <= 0.5f ? kXm : 0) | (fabsf(q.uxp) <= 0.5f ? kXp : 0) |
                               (fabsf(q.uym) <= 0.5f ? kYm : 0) | (fabsf(q.uyp) <= 0.5f ? kYp : 0);
                }
                const float big = fmaxf(aa, bb), small = fminf(aa, bb);
                const float far = fmaxf(fmaxf(fabsf(rx), fabsf(ry)), fabsf(z1) + fabsf(dz) * (float)nz);
                const float err = 2.4e-7f * (fabsf(z1) + zmax);
                // slopes and offsets below 1e4 in every row: margin 0.02; below
                // 1e5: 0.12, row by row
                const bool near = 1e4f * fminf(small, zmin - err) >= fmaxf(big, zmax + err) && far < 1e4f;
                const float L = near ? 1e4f : 1e5f;
                q.half = near ? 0.52f : 0.62f;
                q.t0 = 0.0f; q.k = 3.0e38f;             // no reach: every row is evaluated
                q.cmin = big / L; q.cmax = L * small;
                if (skip && L * small >= big && far < L && big > 1e-3f) {
                    const float d2 = q.a * q.a + q.b * q.b;
                    q.t0 = -__fdividef(q.a * rx + q.b * ry, d2);
                    q.k = 0.88f * rsqrtf(d2);
                    if (zmin - err >= q.cmin && zmax + err <= q.cmax) {
                        q.flags |= kRowsSafe;
                        // the rays of the whole column miss
                        if (fabsf(q.a * ry - q.b * rx) > q.half * (aa + bb)) ok = false;
                        const int in = q.flags & (kXm | kXp | kYm | kYp);
                        if (__popc(in) == 2 && big > 1.2f * (zmax + err)) {
                            // the two faces in the order they are tested
                            const bool xf = q.flags & kXFirst;
                            const int order = xf ? in : (in >> 2) | ((in & 3) << 2);
                            const int f1 = __ffs(order) - 1, f2 = 31 - __clz(order);
                            const float uxm = q.uxm, uxp = q.uxp, uym = q.uym, uyp = q.uyp;
                            auto face = [&](int f, float& d, float& i, float& o, float& h, float& px,
                                            float& py) {
                                const bool x = (f < 2) == xf, m = !(f & 1);
                                d = x ? q.a : q.b; i = fdiv(1.0f, d); o = x ? rx : ry;
                                h = m ? -0.5f : 0.5f;
                                px = x ? h : (m ? uym : uyp);
                                py = x ? (m ? uxm : uxp) : h;
                            };
                            face(f1, q.d1, q.i1, q.o1, q.h1, q.p1x, q.p1y);
                            face(f2, q.d2, q.i2, q.o2, q.h2, q.p2x, q.p2y);
                            const float ex = fsub(q.p2x, q.p1x), ey = fsub(q.p2y, q.p1y);
                            q.e2 = fadd(fmul(ex, ex), fmul(ey, ey));
                            q.flags |= kTwo;
                        }
                    }
                }
                q.ia = ia;
                cols[wp][lane] = q;
            }
            const unsigned mask = __ballot_sync(gm, ok) >> g0;
            __syncwarp(gm);
#pragma unroll 1
            for (int k = 0; k < ZL >> lg; k++) {
                const int wide = __shfl_sync(gm, amax - amin + 1, g0 + v0 + k);
                const int ivk = __shfl_sync(gm, iv, g0 + v0 + k);
                const int ak = __shfl_sync(gm, amin, g0 + v0 + k);
                const unsigned todo = (mask >> (k << lg)) & (0xffffffffu >> (32 - W));
                if ((!todo && wide <= W) || !on) continue;
                const float c = cos_phi[ivk], s = sin_phi[ivk];
                const float xr = fadd(fmul(c, xc), fmul(s, yc));
                const float x1 = fmul(c, -SO), y1 = fmul(s, -SO), z1 = sdz[ivk];
                const float rx = fsub(x1, xc), ry = fsub(y1, yc), rz = fsub(z1, zc);
                const float g = fdiv(SD, fmul(fadd(xr, SO), dz_det));
                int bmax = (int)floorf(fadd(fmul(fadd(zc, dwin), g), (float)nb2));
                int bmin = (int)floorf(fadd(fmul(fsub(zc, dwin), g), (float)nb2));
                bmin = max(bmin, 0); bmax = min(bmax, nb - 1);
                const float* yv = Y + ivk * nd;
                // rows within the columns' reach (uniform rows with safe
                // directions only; 0.03 of a row to spare for the estimate
                // and the 0.005 that plan creation allows from uniform, and the
                // rounding of c)
                if (rows_uniform && wide <= W) {
                    float lo = 3.0e38f, hi = -3.0e38f;
                    for (unsigned t = todo; t; t &= t - 1) {
                        const ChordCol& q = cols[wp][g0 + (k << lg) + __ffs(t) - 1];
                        const float mid = __fdividef(-rz, q.t0);
                        const float d = __fdividef(fmaf(fabsf(mid), q.k, q.half), q.t0 - q.k);
                        if (!(q.flags & kRowsSafe) || !(q.t0 > 2.0f * q.k)) { lo = -3.0e38f; hi = 3.0e38f; }
                        else { lo = fminf(lo, mid - d); hi = fmaxf(hi, mid + d); }
                    }
                    const float e1 = (lo - dv0) * inv_dv, e2 = (hi - dv0) * inv_dv;
                    const float more = 0.03f + 5e-7f * (fabsf(z1) + zmax) * fabsf(inv_dv);
                    bmin = max(bmin, (int)fmaxf(ceilf(fminf(e1, e2) - more), -1.0f));
                    bmax = min(bmax, (int)fminf(floorf(fmaxf(e1, e2) + more), (float)nb));
                }
                for (int ib = bmin; ib <= bmax; ib++) {
                    const float z2 = fadd(__ldg(zdet + ib), z1);
                    const float cz = fsub(z2, z1);
                    const float* yb = yv + (RF ? (long long)ib : (long long)ib * na);
                    if (wide > W) {                     // more columns than lanes: one by one
                        const float cOD = fmul(c, OD), sOD = fmul(s, OD);
                        for (int ia2 = ak; ia2 < ak + wide; ia2++) {
                            const float u = __ldg(ydet + ia2);
                            const float l = chord_box(x1, y1, z1, fsub(cOD, fmul(s, u)),
                                                      fadd(sOD, fmul(c, u)), z2, 1.0f, 1.0f, 1.0f,
                                                      xc, yc, zc);
                            acc = fadd(acc, fmul(l, __ldg(yb + (RF ? (long long)ia2 * nb : (long long)ia2))));
                        }
                        continue;
                    }
                    const float ac = fabsf(cz);
#pragma unroll 1
                    for (unsigned t = todo; t; t &= t - 1) {
                        const ChordCol& q = cols[wp][g0 + (k << lg) + __ffs(t) - 1];
                        if (!(q.flags & kTwo) && ac >= q.cmin && ac <= q.cmax &&
                            fabsf(fmaf(cz, q.t0, rz)) > fmaf(ac, q.k, q.half)) continue;
                        const float l =
                            (q.flags & kTwo) ? chord_two(q, cz, rx, ry, rz)
                            : (q.flags & kAxis)
                                ? chord_box(x1, y1, z1, q.x2, q.y2, z2, 1.0f, 1.0f, 1.0f, xc, yc, zc)
                                : chord_box_col(q, cz, rx, ry, rz);
                        acc = fadd(acc, fmul(l, __ldg(yb + (RF ? (long long)q.ia * nb : (long long)q.ia))));
                    }
                }
            }
        }
    }
    if (on) x[(long long)it * nx * ny * nz + ((long long)iz * ny + iy) * nx + ix] = fmul(acc, scale);
}

// ---------------------------------------------------------------------------
// Dominant-axis forward (version 1): Ax_cone_mf_cpu_new.cpp:23-235 and
// Ax_fan_mf_cpu_new.cpp:18-122. Per slab of the dominant axis the ray touches
// at most two cells along the other in-plane axis and two along z; the case
// analysis (11, 12, 21, 22) and every float operation follow the reference.
// ---------------------------------------------------------------------------
// The up to three cells of one slab: along the other in-plane axis the ray goes
// from cell c1 to c2 (crossing at the fraction rs of the slab; 1 if c2 == c1),
// along z from k1 to k2 (rz). Cells and weights in the order they are met:
// (c1, k1) min(rs, rz); then whichever crossing comes first, |rs - rz|; then (c2,
// k2) 1 - max(rs, rz). These are the reference's cases 11 (the first alone), 12
// and 21 (the first two) and 22 (all three) with their expressions: 1 - rz is rs
// - rz at rs = 1, and a weight of 1 leaves l as it is. A weight of 0 (a slab that
// ends exactly on a plane) still reads its cell, which may not be finite.
__device__ __forceinline__ float gao_slab(float acc, float p1, float p2, float q1, float q2,
                                          float l, int ns, int nz, const float* __restrict__ x,
                                          int ss, int zs, int base)
{
    const int c1 = (int)floorf(p1), c2 = (int)floorf(p2);
    const int k1 = (int)floorf(q1), k2 = (int)floorf(q2);
    const bool dc = c2 != c1, dk = k2 != k1;
    if (c1 < (dc ? -1 : 0) || c1 > ns - 1 || k1 < (dk ? -1 : 0) || k1 > nz - 1) return acc;
    float rs = 1.0f, rz = 1.0f;
    if (dc) rs = fdiv(fsub((float)c2, p1), fsub(p2, p1));
    if (dk) rz = fdiv(fsub((float)k2, q1), fsub(q2, q1));
    const bool zfirst = !dc || rs > rz;             // the z crossing comes first, or alone
    const bool t1 = c1 > -1 && k1 > -1;
    const bool t2 = (dc || dk) && (zfirst ? c1 > -1 && k2 < nz : c2 < ns && k1 > -1);
    const bool t3 = dc && dk && c2 < ns && k2 < nz;
    float x1 = 0.0f, x2 = 0.0f, x3 = 0.0f;
    if (t1) x1 = __ldg(x + (k1 * zs + c1 * ss + base));
    if (t2) x2 = __ldg(x + ((zfirst ? k2 : k1) * zs + (zfirst ? c1 : c2) * ss + base));
    if (t3) x3 = __ldg(x + (k2 * zs + c2 * ss + base));   // < 2^31 (plan creation)
    if (t1) acc = fadd(acc, fmul(fmul(zfirst ? rz : rs, l), x1));
    if (t2) acc = fadd(acc, fmul(fmul(zfirst ? fsub(rs, rz) : fsub(rz, rs), l), x2));
    if (t3) acc = fadd(acc, fmul(fmul(fsub(1.0f, zfirst ? rs : rz), l), x3));
    return acc;
}

// Slabs [lo, hi] of n along which a coordinate that runs from v0 by slope per
// slab can lie in [-1, cells) (one slab and half a cell to spare, and the
// rounding of the reference's expressions, whose terms are below `big`).
__device__ __forceinline__ void slab_range(float v0, float slope, int cells, float big, float& lo,
                                           float& hi)
{
    const float more = 0.5f + 1e-6f * big;
    const float a = __fdividef(-1.0f - more - v0, slope), b = __fdividef((float)cells + more - v0, slope);
    if (fabsf(slope) * 1e6f < 1.0f) {               // parallel: all slabs or none
        const float drift = fabsf(slope) * fmaxf(fabsf(lo), fabsf(hi));
        if (v0 < -1.0f - more - drift || v0 > (float)cells + more + drift) hi = lo - 1.0f;
        return;
    }
    lo = fmaxf(lo, fminf(a, b) - 1.0f);
    hi = fminf(hi, fmaxf(a, b) + 1.0f);
}

// Bound: issue (81 %). 128^3, 120 views, 192 x 160 panel: 3.88 ms with the four
// cases as branches and three divisions per slab, 2.76 with the cells of a slab
// as predicated terms, their loads together, divisions by reciprocals and the
// slabs limited to those the volume can hold, 2.28 with 32-bit indices. 200^3,
// 40 views: 7.26 -> 4.30.
__global__ void __launch_bounds__(128)
k_ref_cone_gao(const float* __restrict__ X, float* __restrict__ y, float* __restrict__ ynorm,
               const float* __restrict__ cphi_v, const float* __restrict__ sphi_v,
               const float* __restrict__ sdz, const float* __restrict__ ydet,
               const float* __restrict__ zdet, const int* __restrict__ vframe, float SO,
               float OD, float scale, int nx, int ny, int nz, float dz, int na, int nb,
               long long nper)
{
    const int ia = blockIdx.x * blockDim.x + threadIdx.x;
    const int ib = blockIdx.y, iv = blockIdx.z;
    if (ia >= na) return;
    const float* x = X + (long long)vframe[iv] * nper;
    const int nx2 = nx / 2, ny2 = ny / 2, nz2 = nz / 2;
    const float c = cphi_v[iv], s = sphi_v[iv];
    const float x1 = fmul(c, -SO), y1 = fmul(s, -SO), z1 = sdz[iv];
    const float u = ydet[ia];
    const float x2 = fsub(fmul(c, OD), fmul(s, u));
    const float y2 = fadd(fmul(s, OD), fmul(c, u));
    const float z2 = fadd(zdet[ib], sdz[iv]);
    // norm3 (Ax_cone_mf_cpu_new.cpp:19-20): double sqrt of float differences, returned as float
    const double ex = (double)fsub(x1, x2), ey = (double)fsub(y1, y2), ez = (double)fsub(z1, z2);
    const float norm = fmul(__double2float_rn(__dsqrt_rn(
                                __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez)))),
                            scale);
    const float tmp = fadd(fmul(fsub(x1, x2), fsub(x1, x2)), fmul(fsub(y1, y2), fsub(y1, y2)));
    const float zz = fmul(fsub(z1, z2), fsub(z1, z2));
    const int zs = nx * ny;
    float acc = 0.0f;
    const bool xdom = fabs_ref(fsub(x1, x2)) > fabs_ref(fsub(y1, y2));
    // primary axis a (walked), secondary in-plane axis b
    const float pa = xdom ? x1 : y1, pb = xdom ? y1 : x1;
    const float s1 = xdom ? fdiv(fsub(y2, y1), fsub(x2, x1)) : fdiv(fsub(x2, x1), fsub(y2, y1));
    const float s2 = xdom ? fdiv(fsub(z2, z1), fsub(x2, x1)) : fdiv(fsub(z2, z1), fsub(y2, y1));
    const int np = xdom ? nx : ny, np2 = xdom ? nx2 : ny2;
    const int ns = xdom ? ny : nx, ns2 = xdom ? ny2 : nx2;
    const int ss = xdom ? nx : 1;
    // the slabs whose cells the volume can hold
    float first = 0.0f, last_ = (float)(np - 1);
    slab_range(pb + s1 * ((float)-np2 - pa) + (float)ns2, s1, ns, fabsf(pb) + fabsf(s1 * pa) + fabsf(s1) * np + ns, first, last_);
    slab_range((z1 + s2 * ((float)-np2 - pa)) / dz + (float)nz2, s2 / dz, nz,
               (fabsf(z1) + fabsf(s2 * pa) + fabsf(s2) * np) / dz + nz, first, last_);
    const int i0 = (int)fmaxf(first, 0.0f), i1 = (int)fminf(last_, (float)(np - 1));
    // divisions by dz and tmp, the same in every slab: by their reciprocals
    const float idz = fdiv(1.0f, dz), itmp = fdiv(1.0f, tmp);
    const float len2 = fadd(tmp, zz);
    // (div_by's remainders must not underflow: nz >= 2, so that a tiny height
    // vanishes in the sum with nz2, and ordinary magnitudes)
    const bool by_recip = nz2 >= 1 && dz > 1e-15f && dz < 1e15f && tmp > 1e-15f && len2 < 1e15f;
    for (int ip = i0; ip <= i1; ip++) {
        const float a1 = (float)(ip - np2), a2 = fadd(a1, 1.0f);
        const float lo = (s1 >= 0.0f) ? a1 : a2, hi = (s1 >= 0.0f) ? a2 : a1;
        const float p1 = fadd(fadd(pb, fmul(s1, fsub(lo, pa))), (float)ns2);
        const float p2 = fadd(fadd(pb, fmul(s1, fsub(hi, pa))), (float)ns2);
        const float zlo = (s2 >= 0.0f) ? a1 : a2, zhi = (s2 >= 0.0f) ? a2 : a1;
        const float w1 = fadd(z1, fmul(s2, fsub(zlo, pa))), w2 = fadd(z1, fmul(s2, fsub(zhi, pa)));
        const float q1 = fadd(by_recip ? div_by(w1, dz, idz) : fdiv(w1, dz), (float)nz2);
        const float q2 = fadd(by_recip ? div_by(w2, dz, idz) : fdiv(w2, dz), (float)nz2);
        const float d = fsub(p2, p1), m = fmul(fadd(fmul(d, d), 1.0f), len2);
        const float l = fsqrt(by_recip ? div_by(m, tmp, itmp) : fdiv(m, tmp));
        acc = gao_slab(acc, p1, p2, q1, q2, l, ns, nz, x, ss, zs, xdom ? ip : ip * nx);
    }
    const long long r = ((long long)iv * nb + ib) * na + ia;
    const float out = fmul(acc, scale);
    y[r] = out;
    if (ynorm) ynorm[r] = fdiv(out, norm);
}

__global__ void __launch_bounds__(128)
k_ref_fan_gao(const float* __restrict__ X, float* __restrict__ y,
              const float* __restrict__ cphi_v, const float* __restrict__ sphi_v,
              const float* __restrict__ ydet, const int* __restrict__ vframe, float SO, float OD,
              float scale, int nx, int ny, int nd, long long nper)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.y;
    if (id >= nd) return;
    const float* x = X + (long long)vframe[iv] * nper;
    const int nx2 = nx / 2, ny2 = ny / 2;
    const float c = cphi_v[iv], s = sphi_v[iv];
    const float x1 = fmul(c, -SO), y1 = fmul(s, -SO);
    const float u = ydet[id];
    const float x2 = fsub(fmul(c, OD), fmul(s, u));
    const float y2 = fadd(fmul(s, OD), fmul(c, u));
    const bool xdom = fabs_ref(fsub(x1, x2)) > fabs_ref(fsub(y1, y2));
    const float sl = xdom ? fdiv(fsub(y2, y1), fsub(x2, x1)) : fdiv(fsub(x2, x1), fsub(y2, y1));
    const float pa = xdom ? x1 : y1, pb = xdom ? y1 : x1;
    const int np = xdom ? nx : ny, np2 = xdom ? nx2 : ny2;
    const int ns = xdom ? ny : nx, ns2 = xdom ? ny2 : nx2;
    float acc = 0.0f;
    for (int ip = 0; ip < np; ip++) {
        const float a1 = (float)(ip - np2), a2 = fadd(a1, 1.0f);
        const float lo = (sl >= 0.0f) ? a1 : a2, hi = (sl >= 0.0f) ? a2 : a1;
        const float p1 = fadd(fadd(pb, fmul(sl, fsub(lo, pa))), (float)ns2);
        const float p2 = fadd(fadd(pb, fmul(sl, fsub(hi, pa))), (float)ns2);
        const int c1 = (int)floorf(p1), c2 = (int)floorf(p2);
#define PIX(cc) __ldg(xdom ? x + (long long)(cc) * nx + ip : x + (long long)ip * nx + (cc))
        const float d = fsub(p2, p1);
        const float l = fsqrt(fadd(fmul(d, d), 1.0f));
        if (c2 == c1) {
            if (c1 >= 0 && c1 <= ns - 1) acc = fadd(acc, fmul(l, PIX(c1)));
        } else if (c2 > 0 && c2 < ns) {
            // the reference reads x outside the image when the two crossings round
            // more than a pixel apart (c1 < 0, Ax_fan_mf_cpu_new.cpp:60-63): skipped
            if (c1 >= 0) acc = fadd(acc, fmul(fmul(fdiv(fsub((float)c2, p1), d), l), PIX(c1)));
            acc = fadd(acc, fmul(fmul(fdiv(fsub(p2, (float)c2), d), l), PIX(c2)));
        } else {
            if (c2 == 0) acc = fadd(acc, fmul(fmul(fdiv(fsub(p2, (float)c2), d), l), PIX(c2)));
            // the reference tests c2 == ny on both branches (Ax_fan_mf_cpu_new.cpp:70,111)
            if (c2 == ny && c1 >= 0 && c1 < ns)
                acc = fadd(acc, fmul(fmul(fdiv(fsub((float)c2, p1), d), l), PIX(c1)));
        }
#undef PIX
    }
    y[(long long)iv * nd + id] = fmul(acc, scale);
}

// ---------------------------------------------------------------------------
// Finite-size beam fan pair (version 2): Ax_fan_mf_cpu_new_fb.cpp:19-123,
// Atx_fan_mf_cpu_new_fb.cpp:20-66, find_area.cpp:18-70.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float edge_area(float a, float b, float c, float x, float y, int& sgn)
{
    const float aa = fabs_ref(a), bb = fabs_ref(b);
    const float hx = fdiv(aa, 2.0f), hy = fdiv(bb, 2.0f);
    const float reach = fadd(hx, hy);
    const float off = fsub(fsub(c, fmul(a, x)), fmul(b, y));
    const float d = fabs_ref(off);
    sgn = off > 0.0f ? 1 : -1;
    if (!(d < reach)) return 0.5f;
    const float flat = fabs_ref(fsub(hx, hy));
    const float inv = (hx < hy) ? fdiv(1.0f, bb) : fdiv(1.0f, aa);
    if (d <= flat) return fmul(d, inv);
    const float r = fsub(reach, d);
    return fsub(0.5f, fdiv(fmul(fmul(0.5f, r), r), fmul(aa, bb)));
}

__device__ __forceinline__ float beam_area(float a1, float b1, float c1, float a2, float b2,
                                           float c2, float x, float y)
{
    int s1, s2;
    const float A1 = edge_area(a1, b1, c1, x, y, s1);
    const float A2 = edge_area(a2, b2, c2, x, y, s2);
    return fabs_ref(fsub(A1, fmul((float)(s1 * s2), A2)));
}

// edges: per (view, bin, edge e) the beam-edge line (Px, Py, Pd), evaluated on
// the host with the float libm calls the reference makes.
__global__ void __launch_bounds__(128)
k_ref_fan_fb(const float* __restrict__ X, float* __restrict__ y,
             const float* __restrict__ cphi_v, const float* __restrict__ sphi_v,
             const float* __restrict__ ydet, const float* __restrict__ edges,
             const int* __restrict__ vframe, float SO, float OD, float scale, float dy_det,
             int nx, int ny, int nd, long long nper)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.y;
    if (id >= nd) return;
    const float* x = X + (long long)vframe[iv] * nper;
    const int nx2 = nx / 2, ny2 = ny / 2;
    const float c = cphi_v[iv], s = sphi_v[iv];
    const float x1 = fmul(c, -SO), y1 = fmul(s, -SO);
    const float hd = fdiv(dy_det, 2.0f);
    const float u0 = fsub(ydet[id], hd), u1 = fadd(ydet[id], hd);
    const float x20 = fsub(fmul(c, OD), fmul(s, u0)), y20 = fadd(fmul(s, OD), fmul(c, u0));
    const float x21 = fsub(fmul(c, OD), fmul(s, u1)), y21 = fadd(fmul(s, OD), fmul(c, u1));
    const float* E = edges + ((long long)iv * nd + id) * 6;
    const float Px0 = E[0], Py0 = E[1], Pd0 = E[2], Px1 = E[3], Py1 = E[4], Pd1 = E[5];
    const bool xdom = fabs_ref(fsub(x1, fdiv(fadd(x20, x21), 2.0f))) >
                      fabs_ref(fsub(y1, fdiv(fadd(y20, y21), 2.0f)));
    const float p1 = xdom ? x1 : y1, q1 = xdom ? y1 : x1;
    const float pe0 = xdom ? x20 : y20, pe1 = xdom ? x21 : y21;
    const float qe0 = xdom ? y20 : x20, qe1 = xdom ? y21 : x21;
    const int np = xdom ? nx : ny, nq = xdom ? ny : nx;
    const int np2 = xdom ? nx2 : ny2, nq2 = xdom ? ny2 : nx2;
    const bool degen = !(pe0 != p1 && pe1 != p1);
    float s0 = 0.0f, s1 = 0.0f;
    if (!degen) { s0 = fdiv(fsub(qe0, q1), fsub(pe0, p1)); s1 = fdiv(fsub(qe1, q1), fsub(pe1, p1)); }
    float acc = 0.0f;
    for (int ip = 0; ip < np; ip++) {
        const float pc = (float)(ip - np2) + 0.5f;
        const float a1 = (float)(ip - np2), a2 = fadd(a1, 1.0f);
        int qmin, qmax;
        if (degen) {
            if (fabs_ref(fsub(p1, pc)) <= 0.5f) { qmin = 0; qmax = nq - 1; }
            else { qmin = 1; qmax = 0; }
        } else {
            const int c0 = (int)floorf(fadd(fadd(q1, fmul(s0, fsub(a1, p1))), (float)nq2));
            const int c1 = (int)floorf(fadd(fadd(q1, fmul(s0, fsub(a2, p1))), (float)nq2));
            const int c2 = (int)floorf(fadd(fadd(q1, fmul(s1, fsub(a1, p1))), (float)nq2));
            const int c3 = (int)floorf(fadd(fadd(q1, fmul(s1, fsub(a2, p1))), (float)nq2));
            qmin = nq - 1; qmax = 0;
            // only in-range crossings move the bounds (Ax_fan_mf_cpu_new_fb.cpp:62-67)
            const int cc[4] = {c0, c1, c2, c3};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (cc[k] < qmin && cc[k] >= 0) qmin = cc[k];
                if (cc[k] > qmax && cc[k] <= nq - 1) qmax = cc[k];
            }
        }
        for (int iq = qmin; iq <= qmax; iq++) {
            const float qc = (float)(iq - nq2) + 0.5f;
            const float l = beam_area(Px0, Py0, Pd0, Px1, Py1, Pd1, xdom ? pc : qc, xdom ? qc : pc);
            if (l > 0.0f)
                acc = fadd(acc, fmul(l, __ldg(xdom ? x + (long long)iq * nx + ip
                                                  : x + (long long)ip * nx + iq)));
        }
    }
    y[(long long)iv * nd + id] = fmul(acc, scale);
}

__global__ void __launch_bounds__(128)
k_ref_fan_fb_adj(float* __restrict__ x, const float* __restrict__ Y,
                 const float* __restrict__ cos_phi, const float* __restrict__ sin_phi,
                 const float* __restrict__ cos_e, const float* __restrict__ sin_e,
                 const int* __restrict__ idY, const int* __restrict__ Nv, int tmp_size,
                 float SO, float OD, float scale, float dy_det, int nx, int ny, int nd, int nt)
{
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y, it = blockIdx.z;
    if (ix >= nx) return;
    const int nd2 = nd / 2, nx2 = nx / 2, ny2 = ny / 2;
    const float SD = fadd(SO, OD);
    const float yc = (float)(iy - ny2) + 0.5f, xc = (float)(ix - nx2) + 0.5f;
    float acc = 0.0f;
    const int nvf = Nv[it];
    for (int j = 0; j < nvf; j++) {
        const int iv = idY[it * tmp_size + j];
        const float* yv = Y + (long long)iv * nd;
        const float c = cos_phi[iv], s = sin_phi[iv];
        const float xr = fadd(fmul(c, xc), fmul(s, yc));
        const float yr = fadd(fmul(-s, xc), fmul(c, yc));
        const float g = fdiv(SD, fmul(fadd(xr, SO), dy_det));
        int hi = (int)floorf(fadd(fmul(fadd(yr, 1.0f), g), (float)nd2));
        int lo = (int)floorf(fadd(fmul(fsub(yr, 1.0f), g), (float)nd2));
        lo = max(lo, 0);
        hi = min(hi, nd - 1);
        for (int id = lo; id <= hi; id++) {
            const float sd0 = __ldg(sin_e + id), cd0 = __ldg(cos_e + id);
            const float sd1 = __ldg(sin_e + id + 1), cd1 = __ldg(cos_e + id + 1);
            const float Px0 = -fadd(fmul(sd0, c), fmul(cd0, s));
            const float Py0 = fsub(fmul(cd0, c), fmul(sd0, s));
            const float Pd0 = fmul(SO, sd0);
            const float Px1 = -fadd(fmul(sd1, c), fmul(cd1, s));
            const float Py1 = fsub(fmul(cd1, c), fmul(sd1, s));
            const float Pd1 = fmul(SO, sd1);
            const float l = beam_area(Px0, Py0, Pd0, Px1, Py1, Pd1, xc, yc);
            if (l > 0.0f) acc = fadd(acc, fmul(l, __ldg(yv + id)));
        }
    }
    x[(long long)it * nx * ny + (long long)iy * nx + ix] = fmul(acc, scale);
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers (device pointers, stream-ordered)
// ---------------------------------------------------------------------------
int fl_ref_forward(fl_plan* p, const float* x, float* y, cudaStream_t st)
{
    const fl_scan& s = p->s;
    if (s.nx % 2 || s.ny % 2 || (s.ndim == 3 && s.nz % 2))
        return fl_set_error(FL_ERR_UNSUPPORTED,
                            "Siddon (version 0) needs even nx, ny, nz: the reference's plane "
                            "lists are one entry short for odd sizes");
    long long nper = (long long)s.nx * s.ny * s.nz;
    if (s.ndim == 2) {
        dim3 grid(fl_div_up(s.na, 128), s.nv);
        k_ref_fan_siddon<<<grid, 128, 0, st>>>(x, y, p->d_cphi_f, p->d_sphi_f, p->d_y_det,
                                               p->d_view_frame, s.SO, s.OD, s.scale, s.nx,
                                               s.ny, s.na, nper);
    } else {
        dim3 grid(fl_div_up(s.na, 128), s.nb, s.nv);
        k_ref_cone_siddon<<<grid, 128, 0, st>>>(x, y, p->d_cphi_f, p->d_sphi_f, p->d_sd_z,
                                                p->d_y_det, p->d_z_det, p->d_view_frame, s.SO,
                                                s.OD, s.scale, s.nx, s.ny, s.nz, s.dz, s.na,
                                                s.nb, nper);
    }
    return fl_check_launch("reference Siddon forward");
}

int fl_ref_adjoint(fl_plan* p, const float* y, float* x, cudaStream_t st)
{
    const fl_scan& s = p->s;
    if (s.ndim == 2) {
        dim3 grid(fl_div_up(s.nx, 128), s.ny, s.nt);
        k_ref_fan_chord_adj<<<grid, 128, 0, st>>>(
            x, y, p->d_cos_phi, p->d_sin_phi, p->d_cos_det, p->d_sin_det, p->d_idY, p->d_Nv,
            p->tmp_size, s.SO, s.OD, s.scale, s.dy_det, s.y_os, s.nx, s.ny, s.na, s.nt);
    } else {
        if ((long long)s.nz * s.nt > 65535)
            return fl_set_error(FL_ERR_UNSUPPORTED, "reference backprojector: nz * nt > 65535");
        // scratch of this call: the flag and a rows-fastest copy of y (a warp's lanes
        // then read neighbouring rows). Without it (fl_plan_scratch) they read y as it
        // is, for the same bits (128^3, 120 views, 192 x 160 panel, source at four half
        // widths: 4.58 ms and 4.95 without; 200 views, 512 x 400: 27.3 and 32.6)
        void* w = fl_plan_scratch(p, 256 + (size_t)p->n_rays * sizeof(float), st);
        int* bad = (int*)w;
        float* yt = w ? (float*)((char*)w + 256) : nullptr;
        int e = fl_check_cuda(w ? cudaMemsetAsync(bad, 0, sizeof(int), st)
                                : cudaMemsetAsync(x, 0, (size_t)p->n_vox * sizeof(float), st),
                              "cudaMemsetAsync");
        const dim3 tg(fl_div_up(s.na, 32), fl_div_up(s.nb, 32), s.nv), tb(32, 8);
        if (w) k_ref_prepare<true><<<tg, tb, 0, st>>>(y, yt, s.na, s.nb, bad, 1);
        else k_ref_prepare<false><<<tg, tb, 0, st>>>(y, yt, s.na, s.nb, x, p->n_vox);
        // 16 or 8 lanes per voxel column where that leaves at least a quarter
        // fewer lanes without a voxel
        int lz = 5;
        auto lanes = [&](int l) { return fl_div_up(s.nz, 1 << l) << l; };
        while (lz > 3 && 4 * lanes(lz - 1) <= 3 * lanes(lz)) lz--;
        const int zruns = fl_div_up(s.nz, 1 << lz);
        const dim3 grid(fl_div_up(s.nx, kChordWarps << (5 - lz)), s.ny, zruns * s.nt);
        auto* k = w ? k_ref_cone_chord_adj<true> : k_ref_cone_chord_adj<false>;
        if (!e)
            k<<<grid, kChordWarps * 32, 0, st>>>(
                x, w ? yt : y, bad, p->d_cos_phi, p->d_sin_phi, p->d_sd_z, p->d_y_det, p->d_z_det, p->d_idY,
                p->d_Nv, p->tmp_size, s.SO, s.OD, s.scale, s.dy_det, s.y_os, s.dz_det, s.dz, s.nx,
                s.ny, s.nz, s.na, s.nb, p->zdet_min, p->zdet_max, p->det_kind != -2, p->v0,
                1.0f / p->dv, zruns, lz);
        if (!e) e = fl_check_launch("reference chord backprojection");
        const int f = w ? fl_check_cuda(cudaFreeAsync(w, st), "cudaFreeAsync") : FL_OK;
        return e ? e : f;
    }
    return fl_check_launch("reference chord backprojection");
}

int fl_ref_gao_forward(fl_plan* p, const float* x, float* y, float* ynorm, cudaStream_t st)
{
    const fl_scan& s = p->s;
    long long nper = (long long)s.nx * s.ny * s.nz;
    if (s.ndim == 2) {
        dim3 grid(fl_div_up(s.na, 128), s.nv);
        k_ref_fan_gao<<<grid, 128, 0, st>>>(x, y, p->d_cphi_f, p->d_sphi_f, p->d_y_det,
                                            p->d_view_frame, s.SO, s.OD, s.scale, s.nx, s.ny,
                                            s.na, nper);
        if (ynorm) return fl_set_error(FL_ERR_UNSUPPORTED, "yNorm is a cone-beam output");
    } else {
        dim3 grid(fl_div_up(s.na, 128), s.nb, s.nv);
        k_ref_cone_gao<<<grid, 128, 0, st>>>(x, y, ynorm, p->d_cphi_f, p->d_sphi_f, p->d_sd_z,
                                             p->d_y_det, p->d_z_det, p->d_view_frame, s.SO, s.OD,
                                             s.scale, s.nx, s.ny, s.nz, s.dz, s.na, s.nb, nper);
    }
    return fl_check_launch("reference dominant-axis forward");
}

int fl_ref_fb_forward(fl_plan* p, const float* x, float* y, cudaStream_t st)
{
    const fl_scan& s = p->s;
    if (s.ndim != 2) return fl_set_error(FL_ERR_UNSUPPORTED, "finite-beam model is fan-beam only");
    if (!p->d_fb_edges) return fl_set_error(FL_ERR_INVALID, "finite-beam model needs dy_det > 0");
    dim3 grid(fl_div_up(s.na, 128), s.nv);
    k_ref_fan_fb<<<grid, 128, 0, st>>>(x, y, p->d_cphi_f, p->d_sphi_f, p->d_y_det, p->d_fb_edges,
                                       p->d_view_frame, s.SO, s.OD, s.scale, s.dy_det, s.nx,
                                       s.ny, s.na, (long long)s.nx * s.ny);
    return fl_check_launch("reference finite-beam forward");
}

int fl_ref_fb_adjoint(fl_plan* p, const float* y, float* x, cudaStream_t st)
{
    const fl_scan& s = p->s;
    if (s.ndim != 2) return fl_set_error(FL_ERR_UNSUPPORTED, "finite-beam model is fan-beam only");
    dim3 grid(fl_div_up(s.nx, 128), s.ny, s.nt);
    k_ref_fan_fb_adj<<<grid, 128, 0, st>>>(x, y, p->d_cos_phi, p->d_sin_phi, p->d_cos_det2,
                                           p->d_sin_det2, p->d_idY, p->d_Nv, p->tmp_size, s.SO,
                                           s.OD, s.scale, s.dy_det, s.nx, s.ny, s.na, s.nt);
    return fl_check_launch("reference finite-beam backprojection");
}
