// flat_adjoint.cu -- backprojection of cone plans whose volume has few heights (the
// model and its forward: matched.cu; the forms for other volumes: cone_adjoint.cu,
// refl_adjoint.cu).
#include "fl_common.cuh"
#include "fl_plan.h"
#include "matched_dev.cuh"

namespace {

constexpr int kFlatX = 8, kFlatY = 16;      // columns of a thread block (a warp: 8 x 4)
constexpr int kFlatRefl = 2, kFlatCone = 4; // heights a thread

// A voxel column per thread, with two or four heights: with few heights the
// lanes along z of the other forms mostly have no voxel. The terms of a voxel and
// their order are the same, so the bits are.
// Bound: latency; the rows of neighbouring columns lie apart, so every height
// adds its loads. us with lanes along z and here: 512^2, 360 views, quarter turns with
// the reflection, one height 1448, 594, two 1543, 953; half turn with it, 90 views, one
// 538, 136, four 567, 191; z mirror 512^2, 181 views, one 1153, 581; general 256^2, 181
// views, one 425, 236, three 440, 370. Six heights a thread 5 % slower for up to
// four; four of the half turn with the reflection 28 % at 384^2 x 8.

// Reflection forms (k_adj_refl: images, slots and sums). BL: blocks per SM.
template <typename TX, typename TW, int NR, int BL>
__global__ void __launch_bounds__(kFlatX * kFlatY, BL)
k_adj_refl_flat(TX* __restrict__ X, const TW* __restrict__ yw, const ColEntry* __restrict__ col,
                const AxisEntry* __restrict__ rowz, const ViewEntry* __restrict__ view, DetGrid G,
                int nx, int ny, int nz, int na, int nb, int nv, float dz,
                const int* __restrict__ skip, int xfold)
{
    if (skip && *skip) return;
    constexpr int NI = 2 * NR, TZ = kFlatRefl;
    const ReflGeom g = refl_geom(NR, nv, na, nb);
    const int ix = blockIdx.x * kFlatX + threadIdx.x % kFlatX;
    const int iy = blockIdx.y * kFlatY + threadIdx.x / kFlatX;
    const int nzw = nz / 2, hx = nx / 2, hy = ny / 2, nbh = g.nbh;
    const int z0 = blockIdx.z * TZ, nk = min(TZ, nzw - z0);
    if (ix >= hx || iy >= hy || (NR == 4 && ix > iy)) return;
    const bool diag = NR == 4 && ix == iy;
    float2 P[TZ][NR], Q[TZ][NR];
#pragma unroll
    for (int z = 0; z < TZ; z++)
#pragma unroll
        for (int j = 0; j < NR; j++) { P[z][j] = make_float2(0.0f, 0.0f); Q[z][j] = P[z][j]; }
    auto trade = [&]() {                                // P and Q
#pragma unroll
        for (int z = 0; z < TZ; z++)
#pragma unroll
            for (int j = 0; j < NR; j++) { const float2 t = P[z][j]; P[z][j] = Q[z][j]; Q[z][j] = t; }
    };
    const float inv_dv = 1.0f / G.dv, vb = G.v0 * inv_dv;
    for (int w = 0; w <= g.ov; w++) {
        int vt, alim;
        long long base;
        refl_view(g, w, vt, base, alim);
        const ViewEntry ve = view[vt];
        const ColEntry* cv = col + (long long)vt * na;
        const AxisEntry* rv = rowz + (long long)vt * nb;
        const TW* yv = yw + base;
        const float zb = -(float)(nz / 2) * dz - ve.sz;
#pragma unroll 1
        for (int k = 0; k < (diag ? NR : NI); k++) {
            if (k == NR) trade();                       // the D images
            int px, py, alo, ahi;
            float dmin, dmax;
            refl_column<NR>(k, ix, iy, nx, ny, px, py);
            column_window(G, ve.c, ve.s, (float)(px - hx), (float)(py - hy), 1.0f, 1.0f, na, alo,
                          ahi, dmin, dmax);
            ahi = min(ahi, alim - 1);
            for (int ia = alo; ia <= ahi; ia++) {
                if (!FL_IN(ia, na)) continue;
                float bh, be, l, h;
                if (!cone_column(cv[ia], px, py, nx, ny, bh, be, l, h)) continue;
                const float r1 = __fdividef(inv_dv, __fadd_rn(bh, l) + ve.ac);
                const float r2 = __fdividef(inv_dv, __fadd_rn(bh, h) + ve.ac);
                const float s1 = dz * r1, c1 = zb * r1 - vb - 0.02f;
                const float s2 = dz * r2, c2 = zb * r2 - vb + 0.02f;
                const TW* yt = yv + (long long)NI * nbh * ia;
#pragma unroll
                for (int z = 0; z < TZ; z++) {
                    if (z >= nk) break;
                    const float fz = (float)(z0 + z), fz1 = (float)(z0 + z + 1);
                    const int blo = max(__float2int_ru(fmaf(fz, s1, c1)), 0);
                    const int bhi = min(__float2int_rd(fmaf(fz1, s2, c2)), nbh - 1);
#pragma unroll 1
                    for (int ib = blo; ib <= bhi; ib++) {
                        if (!FL_IN(ib, nbh)) continue;
                        const float2 az = row_planes(rv[ib], fz, fz1, bh, be);
                        float t[NI], u[NI];
                        ld_in<TW, NI>(yt + NI * ib, t);
                        ld_in<TW, NI>(yt + g.plane + NI * ib, u);
                        const float wgt = fminf(h, az.x) - fmaxf(l, az.y);
                        if (wgt > 0.0f) {
                            const float2 w2 = make_float2(wgt, wgt);
#pragma unroll
                            for (int j = 0; j < NR; j++) {
                                P[z][j] = __ffma2_rn(w2, make_float2(t[2 * j], t[2 * j + 1]), P[z][j]);
                                Q[z][j] = __ffma2_rn(w2, make_float2(u[2 * j], u[2 * j + 1]), Q[z][j]);
                            }
                        }
                    }
                }
            }
            // next image: P rotates back one place, Q forward one
#pragma unroll
            for (int z = 0; z < TZ; z++) {
                const float2 a = P[z][0];
#pragma unroll
                for (int j = 0; j + 1 < NR; j++) P[z][j] = P[z][j + 1];
                P[z][NR - 1] = a;
                const float2 b = Q[z][NR - 1];
#pragma unroll
                for (int j = NR - 1; j > 0; j--) Q[z][j] = Q[z][j - 1];
                Q[z][0] = b;
            }
        }
        if (!diag) trade();                             // C sums back into P
    }
    const long long nxy = (long long)nx * ny;
#pragma unroll
    for (int z = 0; z < TZ; z++) {
        if (z >= nk) break;
        const int zl = z0 + z;
#pragma unroll
        for (int j = 0; j < NI; j++) {
            if (diag && j >= NR) continue;
            float2 a = j < NR ? P[z][j % NR] : Q[z][j % NR];
            if (diag) {
                const float2 b = Q[z][(j + 1) % NR];
                a.x += b.x; a.y += b.y;
            }
            int qx, qy;
            refl_column<NR>(j, ix, iy, nx, ny, qx, qy);
            if (xfold) {
                Store<TX>::st2(X + orbit_pair(qx, qy, zl, nx, ny), a.x, a.y);
            } else {
                const long long q = (long long)qy * nx + qx;
                Store<TX>::st(X + zl * nxy + q, a.x);
                Store<TX>::st(X + (nz - 1 - zl) * nxy + q, a.y);
            }
        }
    }
}

// General and (MIRROR) z-mirror forms (k_adj_cone).
template <typename TX, typename TW, bool MIRROR>
__global__ void __launch_bounds__(kFlatX * kFlatY, 8)
k_adj_cone_flat(TX* __restrict__ X, const TW* __restrict__ yw, const ColEntry* __restrict__ col,
                const AxisEntry* __restrict__ rowz, const ViewEntry* __restrict__ view,
                const int* __restrict__ idY, const int* __restrict__ Nv, int tmp_size, DetGrid G,
                int nx, int ny, int nz, int na, int nb, float dz, int zruns,
                const int* __restrict__ skip, int xfold)
{
    if (skip && *skip) return;
    constexpr int V = MIRROR ? 2 : 1, TZ = kFlatCone;
    const int ix = blockIdx.x * kFlatX + threadIdx.x % kFlatX;
    const int iy = blockIdx.y * kFlatY + threadIdx.x / kFlatX;
    const int nzw = MIRROR ? nz / 2 : nz, nbw = MIRROR ? nb / 2 : nb;
    const int z0 = (int)(blockIdx.z % zruns) * TZ, it = blockIdx.z / zruns, nk = min(TZ, nzw - z0);
    if (ix >= nx || iy >= ny) return;
    float2 acc[TZ];                                     // .y: the mirrored voxel
#pragma unroll
    for (int z = 0; z < TZ; z++) acc[z] = make_float2(0.0f, 0.0f);
    const float inv_dv = 1.0f / G.dv, vb = G.v0 * inv_dv;
    const int nvf = Nv[it];
    const int* views = idY + it * tmp_size;
    for (int jv = 0; jv < nvf; jv++) {
        const int iv = views[jv];
        const ViewEntry ve = view[iv];
        int alo, ahi;
        float dmin, dmax;
        column_window(G, ve.c, ve.s, (float)(ix - nx / 2), (float)(iy - ny / 2), 1.0f, 1.0f, na, alo,
                      ahi, dmin, dmax);
        const AxisEntry* rv = rowz + (long long)iv * nb;
        for (int ia = alo; ia <= ahi; ia++) {
            if (!FL_IN(ia, na)) continue;
            const long long ray = (long long)iv * na + ia;
            float bh, be, l, h;
            if (!cone_column(col[ray], ix, iy, nx, ny, bh, be, l, h)) continue;
            const float r1 = __fdividef(inv_dv, __fadd_rn(bh, l) + ve.ac);
            const float r2 = __fdividef(inv_dv, __fadd_rn(bh, h) + ve.ac);
            const TW* yt = yw + (long long)(V * nbw) * ray;
#pragma unroll
            for (int z = 0; z < TZ; z++) {
                if (z >= nk) break;
                const int zl = z0 + z;
                const float za = (float)(zl - nz / 2) * dz - ve.sz, zb = (float)(zl + 1 - nz / 2) * dz - ve.sz;
                const float a1 = za * r1 - vb, b2 = zb * r2 - vb;
                float elo = a1, ehi = b2;
                if (!MIRROR) {                          // (the mirror's rays descend and its rows rise)
                    const float a2 = za * r2 - vb, b1 = zb * r1 - vb;
                    elo = fminf(fminf(a1, a2), fminf(b1, b2));
                    ehi = fmaxf(fmaxf(a1, a2), fmaxf(b1, b2));
                }
                const int blo = max(__float2int_ru(elo - 0.02f), 0);
                const int bhi = min(__float2int_rd(ehi + 0.02f), nbw - 1);
#pragma unroll 1
                for (int ib = blo; ib <= bhi; ib++) {
                    if (!FL_IN(ib, nbw)) continue;
                    float t[V];
                    ld_in<TW, V>(yt + V * ib, t);
                    const float2 az = row_planes(rv[ib], (float)zl, (float)(zl + 1), bh, be);
                    const float lo = MIRROR ? az.y : fminf(az.x, az.y);
                    const float hi = MIRROR ? az.x : fmaxf(az.x, az.y);
                    const float w = fminf(h, hi) - fmaxf(l, lo);
                    if (w > 0.0f) {
                        if (MIRROR) acc[z] = __ffma2_rn(make_float2(w, w), make_float2(t[0], t[V - 1]), acc[z]);
                        else acc[z].x = fmaf(w, t[0], acc[z].x);
                    }
                }
            }
        }
    }
    const long long nxy = (long long)nx * ny, q = (long long)iy * nx + ix;
    TX* xf = X + (long long)it * nxy * nz;
#pragma unroll
    for (int z = 0; z < TZ; z++) {
        if (z >= nk) break;
        const int zl = z0 + z;
        if (MIRROR && xfold) {
            Store<TX>::st2(xf + 2 * (zl * nxy + q), acc[z].x, acc[z].y);
        } else {
            Store<TX>::st(xf + zl * nxy + q, acc[z].x);
            if (MIRROR) Store<TX>::st(xf + (nz - 1 - zl) * nxy + q, acc[z].y);
        }
    }
}

template <typename TX, typename TW>
void launch(fl_plan* p, const void* yw, void* x, const int* skip, int xfold, cudaStream_t st)
{
    const fl_scan& s = p->s;
    if (const int NR = fl_plan_refl(p)) {
        const dim3 g(fl_div_up(s.nx / 2, kFlatX), fl_div_up(s.ny / 2, kFlatY), fl_div_up(s.nz / 2, kFlatRefl));
        // five blocks of the quarter turns' 92 registers per SM, six of 80 where the
        // octant's half of the grid would not fit at once (512^2, 48 views, 8 heights of
        // both halves 175 us with five, 202; 12: 287, 212)
        const bool many = (long long)g.x * g.y * g.z / 2 > 5LL * p->sms;
        auto* k = NR == 2 ? k_adj_refl_flat<TX, TW, 2, 8>
                  : many  ? k_adj_refl_flat<TX, TW, 4, 6> : k_adj_refl_flat<TX, TW, 4, 5>;
        k<<<g, kFlatX * kFlatY, 0, st>>>((TX*)x, (const TW*)yw, p->d_col, p->d_rowz, p->d_view, det_grid(p),
                                         s.nx, s.ny, s.nz, s.na, s.nb, s.nv, s.dz, skip, xfold);
        return;
    }
    const int zruns = fl_div_up(p->zmirror ? s.nz / 2 : s.nz, kFlatCone);
    const dim3 g(fl_div_up(s.nx, kFlatX), fl_div_up(s.ny, kFlatY), zruns * s.nt);
    auto* k = p->zmirror ? k_adj_cone_flat<TX, TW, true> : k_adj_cone_flat<TX, TW, false>;
    k<<<g, kFlatX * kFlatY, 0, st>>>((TX*)x, (const TW*)yw, p->d_col, p->d_rowz, p->d_view, p->d_idY, p->d_Nv,
                                     p->tmp_size, det_grid(p), s.nx, s.ny, s.nz, s.na, s.nb, s.dz, zruns, skip,
                                     p->zmirror ? xfold : 0);
}

}  // namespace

// Heights (of the half volume with the z mirror) up to which a column per thread is
// faster, by the image's size: the lanes along z want columns, too, to fill the GPU
// (us, lanes along z and a column per thread; general 128^2, 181 views, one height 264,
// 211, two 248, 284; 192^2, 45 views, three 98, 90, four 98, 109; 384^2 six 300, 285;
// 512^2 six 480, 471; half turn with the reflection, 90 views, 192^2 one 107, 109, two
// 112, 154; 256^2 three 168, 158, four 168, 170; 512^2 six 465, 452; quarter turns,
// 48 views, 256^2 two 102, 98, six 109, 121; 512^2 four 212, 175). Where the
// runs of all frames are more than a grid's z holds, the lanes' one run per frame fits.
bool fl_plan_adj_flat(const fl_plan* p)
{
    const fl_scan& s = p->s;
    const int NR = fl_plan_refl(p);
    if (s.ndim != 3 || (!NR && p->zmirror && p->rot) || (NR && p->adj_chunks > 1)) return false;
    const int h = p->zmirror ? s.nz / 2 : s.nz;
    const long long area = (long long)s.nx * s.ny * s.nt / (NR ? 2 : 1);
    if ((long long)fl_div_up(h, NR ? kFlatRefl : kFlatCone) * s.nt > 65535) return false;
    return area >= (1 << 14) && h <= (area < (1 << 15) ? 1 : area < (1 << 16) ? 3 : 6);
}

void fl_matched_adjoint_flat(fl_plan* p, const void* yw, int wt, void* x, int xt, const int* skip,
                             int xfold, cudaStream_t st)
{
    if (wt == FL_F32) {
        if (xt == FL_F32) launch<float, float>(p, yw, x, skip, xfold, st);
        else if (xt == FL_F16) launch<__half, float>(p, yw, x, skip, xfold, st);
        else launch<__nv_bfloat16, float>(p, yw, x, skip, xfold, st);
    } else {
        if (xt == FL_F32) launch<float, __half>(p, yw, x, skip, xfold, st);
        else if (xt == FL_F16) launch<__half, __half>(p, yw, x, skip, xfold, st);
        else launch<__nv_bfloat16, __half>(p, yw, x, skip, xfold, st);
    }
}

FL_OOB_ACCESSOR(fl_oob_flat)
