// cone_adjoint.cu -- backprojection of the cone plans' general and z-mirror
// forms (the model and its forward: matched.cu; the reflection forms:
// refl_adjoint.cu).
#include "fl_common.cuh"
#include "fl_plan.h"
#include "matched_dev.cuh"

namespace {

// A candidate: one detector column of one view whose rays can cross a warp's
// block of voxel columns.
template <int NP>
struct alignas(16) ConeCand {
    float bh, be;                  // frame (anchor)
    float r1, r2;                  // rows per unit of height at the block's near and far end
    float sz;                      // source z
    unsigned ray;                  // iv na + ia
    int view, pad;
    float2 lh[NP == 1 ? 2 : NP];   // entry and exit of the block's columns (l >= h: missed)
};

constexpr int kConeWarps = 4;      // 2 x 2 blocks of columns per thread block

// General and (MIRROR) z-mirror backprojection. A warp owns a PB x PB block of
// voxel columns of one frame and 32 neighbouring heights, a voxel of each column
// per lane (MIRROR: of the lower half, with its mirror; yw then holds pairs).
// For up to 32 views at a time the lanes find the views' detector windows of
// the block (a view whose rows miss the warp's heights has none); then they
// take the windows' detector columns, several views together, one candidate per
// lane: the rays' crossings with the block's columns, kept in shared memory.
// Every lane then visits the candidates in order (views in the frame's order,
// columns in increasing order) and the detector rows that can meet its voxels,
// evaluating w_rV as the forward walk does. A row's value is loaded once for
// the block's columns, and neighbouring lanes load neighbouring rows.
// lanes: log2 of the lanes per block (5 .. 2), a constant 5 with FULL.
// Bound: issue and latency. The form before it (one thread per column and run
// of 8 voxels, its own column set-up per view) issued 90 warp instructions per
// useful weight of a circular scan and 183 of a helix, whose views mostly miss a
// run: 151 x 151 x 97, 211 views 4.42 ms, 255^3 / 179 views 24.8, helix 128^3 /
// 241 views 2.07, mirror 152 x 152 x 98 / 211 views 1.92, 47 x 47 x 33 / 61
// views 0.41. With one column per warp 3.51, 23.4, 1.42, 1.86, 0.08; 2 x 2
// columns: 2.30, 15.2, 0.92, 1.33, 0.085. 8 blocks per SM against 7: mirror
// 1.40; 10: 2.53 and 16.4 on the first two.
template <typename TX, int PB, typename TW, bool MIRROR, bool FULL>
__global__ void __launch_bounds__(kConeWarps * 32, 7)
k_adj_cone(TX* __restrict__ X, const TW* __restrict__ yw, const ColEntry* __restrict__ col,
           const AxisEntry* __restrict__ rowz, const ViewEntry* __restrict__ view,
           const int* __restrict__ idY, const int* __restrict__ Nv, int tmp_size, DetGrid G,
           int nx, int ny, int nz, int na, int nb, float dz, int zruns,
           const int* __restrict__ skip, int xfold, int lanes)
{
    if (skip && *skip) return;
    constexpr int NP = PB * PB, V = MIRROR ? 2 : 1;
    const int lz = FULL ? 5 : lanes;
    __shared__ ConeCand<NP> cand[kConeWarps][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int nzw = MIRROR ? nz / 2 : nz, nbw = MIRROR ? nb / 2 : nb;
    // the lane's group of ZL = 2^lz lanes, its first lane and lanes' mask
    const int ZL = 1 << lz, g0 = FULL ? 0 : lane & ~(ZL - 1), sub = lane & (ZL - 1);
    const unsigned gm = FULL ? 0xffffffffu : (0xffffffffu >> (32 - ZL)) << g0;
    const int X0 = PB * (((2 * blockIdx.x + (wp & 1)) << (5 - lz)) + (g0 >> lz));
    const int Y0 = PB * (2 * blockIdx.y + (wp >> 1));
    const int zc = (int)(blockIdx.z % zruns) << lz, it = blockIdx.z / zruns;
    if (X0 >= nx || Y0 >= ny) return;                   // whole groups
    const int z = zc + sub;
    const bool on = z < nzw;
    float2 acc[NP];                                     // .y: the mirrored voxel
#pragma unroll
    for (int c = 0; c < NP; c++) acc[c] = make_float2(0.0f, 0.0f);
    const float inv_dv = 1.0f / G.dv, vb = G.v0 * inv_dv;
    const float fz = (float)z, fz1 = (float)(z + 1);
    const float h0 = (float)(z - nz / 2) * dz, h1 = (float)(z + 1 - nz / 2) * dz;
    const int nvf = Nv[it];
    const int* views = idY + it * tmp_size;
    for (int jb = 0; jb < nvf; jb += ZL) {
        // this lane's view and its window of the block
        int iv = 0, alo = 0, ahi = -1;
        if (jb + sub < nvf) {
            iv = views[jb + sub];
            const ViewEntry ve = view[iv];
            float dmin, dmax;
            // (the part of the block inside the grid: a source beside the grid's
            // corner may stand in the rest)
            column_window(G, ve.c, ve.s, (float)(X0 - nx / 2), (float)(Y0 - ny / 2),
                          (float)min(PB, nx - X0), (float)min(PB, ny - Y0), na, alo, ahi, dmin, dmax);
            // rows of the group's heights at the block's depths, a row to spare
            const float za = (float)(zc - nz / 2) * dz - ve.sz;
            const float zb = (float)(min(zc + ZL, nzw) - nz / 2) * dz - ve.sz;
            const float q1 = G.SD * __fdividef(inv_dv, dmin), q2 = G.SD * __fdividef(inv_dv, dmax);
            const float e1 = za * q1, e2 = za * q2, e3 = zb * q1, e4 = zb * q2;
            if (fmaxf(fmaxf(e1, e2), fmaxf(e3, e4)) - vb < -1.0f ||
                fminf(fminf(e1, e2), fminf(e3, e4)) - vb > (float)nbw) { alo = 0; ahi = -1; }
        }
        const int maxw = __reduce_max_sync(gm, ahi - alo + 1);
        if (maxw <= 0) continue;
        int lg = FULL ? (PB == 1 ? 2 : 3) : min(PB == 1 ? 2 : 3, lz);   // 4 .. ZL candidates per view
        while (lg < lz && (1 << lg) < maxw) lg++;
        const int W = 1 << lg;
        for (int v0 = 0; v0 < min(ZL, nvf - jb); v0 += ZL >> lg) {
            const int vm = g0 + v0 + (sub >> lg);
            const int lo = __shfl_sync(gm, alo, vm), span = __shfl_sync(gm, ahi - alo, vm);
            const int ivm = __shfl_sync(gm, iv, vm);
            for (int j0 = 0; j0 < maxw; j0 += W) {      // once, or W = ZL and one view
                const int j = j0 + (sub & (W - 1)), ia = (int)((unsigned)lo + j);
                bool ok = j <= span && FL_IN(ia, na);   // (lo + j can wrap; not where ok)
                __syncwarp(gm);
                if (ok) {
                    const ColEntry ce = col[(long long)ivm * na + ia];
                    ConeCand<NP>& q = cand[wp][lane];
                    // the frame and the crossings of the block's planes
                    const bool xd = x_dominant(ce.x, ce.y);
                    float bh, be;
                    make_anchor<kSegCone>(xd ? ce.x : ce.y, (xd ? X0 : Y0) >> kSegCone,
                                          xd ? nx : ny, bh, be);
                    const float mx = __fsub_rn((float)X0, ce.x.kq);
                    const float my = __fsub_rn((float)Y0, ce.y.kq);
                    const float cbx = __fsub_rn(ce.x.c, be), cby = __fsub_rn(ce.y.c, be);
                    float tx[PB + 1], ty[PB + 1];
#pragma unroll
                    for (int i = 0; i <= PB; i++) {
                        tx[i] = xrel(ce.x, __fadd_rn(mx, (float)i), bh, cbx);
                        ty[i] = xrel(ce.y, __fadd_rn(my, (float)i), bh, cby);
                    }
                    float lmin = 3.0e38f, hmax = -3.0e38f;
#pragma unroll
                    for (int c = 0; c < NP; c++) {
                        const int i = c % PB, j = c / PB;
                        float l = fmaxf(fminf(tx[i], tx[i + 1]), fminf(ty[j], ty[j + 1]));
                        float h = fminf(fmaxf(tx[i], tx[i + 1]), fmaxf(ty[j], ty[j + 1]));
                        if (X0 + i >= nx || Y0 + j >= ny) { l = 1.0f; h = 0.0f; }
                        q.lh[c] = make_float2(l, h);
                        if (l < h) { lmin = fminf(lmin, l); hmax = fmaxf(hmax, h); }
                    }
                    ok = lmin < hmax;
                    const ViewEntry ve = view[ivm];
                    q.bh = bh; q.be = be;
                    q.r1 = __fdividef(inv_dv, __fadd_rn(bh, lmin) + ve.ac);
                    q.r2 = __fdividef(inv_dv, __fadd_rn(bh, hmax) + ve.ac);
                    q.sz = ve.sz;
                    q.ray = (unsigned)ivm * na + ia; q.view = ivm;
                }
                unsigned todo = __ballot_sync(gm, ok) >> g0;
                if (!FULL && ZL < 32) todo &= (1u << ZL) - 1u;
                __syncwarp(gm);
#pragma unroll 1
                for (; todo; todo &= todo - 1) {
                    const ConeCand<NP>& q = cand[wp][g0 + __ffs(todo) - 1];
                    const float bh = q.bh, be = q.be, za = h0 - q.sz, zb = h1 - q.sz;
                    // rows that are inside the voxel's heights somewhere in the
                    // block: between its planes' crossings at the block's ends
                    const float a1 = za * q.r1 - vb, b2 = zb * q.r2 - vb;
                    float elo = a1, ehi = b2;
                    if (!MIRROR) {                      // (the mirror's rays descend and its rows rise)
                        const float a2 = za * q.r2 - vb, b1 = zb * q.r1 - vb;
                        elo = fminf(fminf(a1, a2), fminf(b1, b2));
                        ehi = fmaxf(fmaxf(a1, a2), fmaxf(b1, b2));
                    }
                    const int blo = max(__float2int_ru(elo - 0.02f), 0);
                    const int bhi = min(__float2int_rd(ehi + 0.02f), on ? nbw - 1 : -1);
                    const AxisEntry* rv = rowz + (long long)q.view * nb;
                    const TW* yt = yw + (long long)(V * nbw) * q.ray;
                    float2 lh[NP];
#pragma unroll
                    for (int c = 0; c < NP; c++) lh[c] = q.lh[c];
#pragma unroll 1
                    for (int ib = blo; ib <= bhi; ib++) {
                        if (!FL_IN(ib, nbw)) continue;
                        const AxisEntry re = rv[ib];
                        float t[V];
                        ld_in<TW, V>(yt + V * ib, t);
                        const float2 az = row_planes(re, fz, fz1, bh, be);
                        const float zl = MIRROR ? az.y : fminf(az.x, az.y);
                        const float zh = MIRROR ? az.x : fmaxf(az.x, az.y);
#pragma unroll
                        for (int c = 0; c < NP; c++) {
                            const float w = fminf(lh[c].y, zh) - fmaxf(lh[c].x, zl);
                            if (w > 0.0f) {
                                if (MIRROR)
                                    acc[c] = __ffma2_rn(make_float2(w, w), make_float2(t[0], t[V - 1]), acc[c]);
                                else
                                    acc[c].x = fmaf(w, t[0], acc[c].x);
                            }
                        }
                    }
                }
            }
        }
    }
    if (!on) return;
    const long long nxy = (long long)nx * ny;
    TX* xf = X + (long long)it * nxy * nz;
#pragma unroll
    for (int c = 0; c < NP; c++) {
        const int ix = X0 + c % PB, iy = Y0 + c / PB;
        if (ix >= nx || iy >= ny) continue;
        const long long q = (long long)iy * nx + ix;
        if (MIRROR && xfold) {
            Store<TX>::st2(xf + 2 * (z * nxy + q), acc[c].x, acc[c].y);
        } else {
            Store<TX>::st(xf + z * nxy + q, acc[c].x);
            if (MIRROR) Store<TX>::st(xf + (nz - 1 - z) * nxy + q, acc[c].y);
        }
    }
}

template <typename TX, typename TW, bool MIRROR>
void launch(fl_plan* p, const void* yw, void* x, const int* skip, int xfold, cudaStream_t st)
{
    const fl_scan& s = p->s;
    const int nzw = MIRROR ? s.nz / 2 : s.nz;
    // as for the reflection form (refl_adjoint.cu): 2 x 2 columns per warp once
    // such warps fill the GPU
    auto warps = [&](int pb, int lz) {
        return ((long long)fl_div_up(s.nx, pb) * fl_div_up(s.ny, pb) * fl_div_up(nzw, 1 << lz) * s.nt) >>
               (5 - lz);
    };
    auto lanes_log2 = [&](int pb) { return adj_lanes_log2(p, nzw, 2, [&](int lz) { return warps(pb, lz); }); };
    const int PB = warps(2, lanes_log2(2)) >= adj_full_warps(p) ? 2 : 1, lz = lanes_log2(PB);
    const int zruns = fl_div_up(nzw, 1 << lz);
    const dim3 grid(fl_div_up(s.nx, (2 * PB) << (5 - lz)), fl_div_up(s.ny, 2 * PB), zruns * s.nt);
    auto* k = PB == 2 ? (lz == 5 ? k_adj_cone<TX, 2, TW, MIRROR, true> : k_adj_cone<TX, 2, TW, MIRROR, false>)
                      : (lz == 5 ? k_adj_cone<TX, 1, TW, MIRROR, true> : k_adj_cone<TX, 1, TW, MIRROR, false>);
    k<<<grid, kConeWarps * 32, 0, st>>>((TX*)x, (const TW*)yw, p->d_col, p->d_rowz, p->d_view, p->d_idY,
                                        p->d_Nv, p->tmp_size, det_grid(p), s.nx, s.ny, s.nz, s.na, s.nb,
                                        s.dz, zruns, skip, xfold, lz);
}

template <typename TX, typename TW>
void launch_form(fl_plan* p, const void* yw, void* x, const int* skip, int xfold, cudaStream_t st)
{
    if (p->zmirror) launch<TX, TW, true>(p, yw, x, skip, xfold, st);
    else launch<TX, TW, false>(p, yw, x, skip, 0, st);
}

}  // namespace

void fl_matched_adjoint_cone(fl_plan* p, const void* yw, int wt, void* x, int xt, const int* skip,
                             int xfold, cudaStream_t st)
{
    if (wt == FL_F32) {
        if (xt == FL_F32) launch_form<float, float>(p, yw, x, skip, xfold, st);
        else if (xt == FL_F16) launch_form<__half, float>(p, yw, x, skip, xfold, st);
        else launch_form<__nv_bfloat16, float>(p, yw, x, skip, xfold, st);
    } else {
        if (xt == FL_F32) launch_form<float, __half>(p, yw, x, skip, xfold, st);
        else if (xt == FL_F16) launch_form<__half, __half>(p, yw, x, skip, xfold, st);
        else launch_form<__nv_bfloat16, __half>(p, yw, x, skip, xfold, st);
    }
}

FL_OOB_ACCESSOR(fl_oob_cone)
