// refl_adjoint.cu -- backprojection of the cone plans' reflection forms (the
// model and its forward: matched.cu).
#include <type_traits>

#include "fl_common.cuh"
#include "fl_plan.h"
#include "matched_dev.cuh"

namespace {

// Lower corner of image k of the PB x PB block of columns at (X0, Y0).
template <int NR, int PB>
__device__ __forceinline__ void refl_corner(int k, int X0, int Y0, int nx, int ny, int& bx,
                                            int& by)
{
    int x1, y1;
    refl_column<NR>(k, X0, Y0, nx, ny, bx, by);
    refl_column<NR>(k, X0 + PB - 1, Y0 + PB - 1, nx, ny, x1, y1);
    bx = min(bx, x1); by = min(by, y1);
}

// A candidate of the backprojection below: one detector column in one image of
// a warp's block of columns.
template <int NP>
struct alignas(16) ReflCand {
    float bh, be;           // frame (anchor)
    float c1, s1, c2, s2;   // detector rows of voxel z: [c1 + s1 z, c2 + s2 (z + 1)]
    int off, pad;           // first orbit of the detector column
    float2 lh[NP == 1 ? 2 : NP];   // entry and exit of the block's columns (l >= h: missed)
};

constexpr int kReflWarps = 4;       // 2 x 2 blocks of columns per thread block

// Reflection + z-mirror backprojections (fl_plan::refl). NR = 4 (quarter
// turns, nx == ny == n): voxel columns V0 = (x, y) of the octant x <= y < n/2;
// NR = 2 (half turn): of the quadrant x < nx/2, y < ny/2. A warp owns a PB x PB
// block of columns; a lane, one voxel of each column's lower half, its mirror
// and the images C_k = S^k V0 and D_k = S^k M V0 (k < NR; for NR = 4 and x ==
// y, D_k = C_{k+3} and only the C_k are visited). The warp visits the walked
// views w = 0 .. ov (refl_view). In view w a weight of column C_k multiplies
// turn slot j (view w + j nv/NR) into C_{k+j} and reflected slot j (view j
// nv/NR - w, column na-1-a) into D_{j-k}; a weight of D_k, turn slot j into
// D_{k+j} and reflected slot j into C_{j-k}. One weight thus feeds 4 NR (voxel,
// ray) pairs. yw is the packed input of k_weight_packed_refl / k_fwd_refl (two
// planes); X the folded volume's orbits (xfold) or the standard one.
// The lanes of a warp share the columns, so they share the detector columns
// and the rays' crossings with them: the lanes find those together (one
// candidate (image, detector column) each) and keep them in shared memory; then
// every lane takes the candidates one after another and visits the detector
// rows that meet its own voxels, neighbours of the next lane's. A row's orbit
// is loaded once for the block's columns.
// Bound: latency, with no unit saturated (256^3, 360 views: L1 data pipe 64.7 %,
// issue 47 %, 16 warps per SM at 128 registers). The form before it gave every
// thread a column of its own and every lane another (72 %, 54 %, 143 warp
// instructions per weight, the column setup repeated in each thread): 10.36 ms
// at 256^3 / 360 views, 152.4 ms at 512^3 / 720, 2.84 ms at 256^3 / 90 (half
// turn), 0.207 ms at 64^3 / 72. Lanes along z with one column per warp: 9.34,
// 140, 2.91, 0.102; 2 x 2 columns: 7.22, 102, 2.11, 0.203; with the views of a
// large input in chunks and vector stores of the packed input: 6.94, 98.7, 2.08,
// 0.100; the row table's pointer held (held): 6.79 at 256^3; NR = 2 with 2 x 2
// columns at 7 blocks per SM (4: 2.04): 1.94 at 256^3 / 90. Slower or no faster:
// two rows per iteration (8.9 ms at 256^3), 3 and 5 blocks per SM (7.5, 10.6),
// blocks of 8 and 16 warps (7.4), even and odd rows kept apart so that the lanes'
// loads are dense (7.26; 108 at 512^3), the next row's table entry loaded ahead
// (7.7), a run-time lane count for FULL (+10 %).
// View chunks: the walked views w0 .. w1 only. A launch that is not the
// first continues the sums it finds in X (FP32, either layout) and one that
// is not the last leaves them there, so a sequence of launches over
// consecutive chunks adds every term in the order one launch would: the bits
// are the same. On the diagonal (NR = 4, x == y) P and Q are carried apart
// between chunks, P in X and Q in dq (dq[((x * dqz + z) * NR + j)] for the
// voxel pair at height z < nz/2), and combined by the last.
// lanes: log2 of the lanes per block of columns (5, 4 or 3; fewer where the
// volume's half height would leave many lanes without a voxel), so a warp takes
// 32 >> lanes blocks side by side; a constant 5 with FULL.
template <typename TX, int PB, typename TW, int NR, bool FULL>
__global__ void __launch_bounds__(kReflWarps * 32, PB == 2 && NR == 4 ? 4 : 7)
k_adj_refl(TX* __restrict__ X, const TW* __restrict__ yw, const ColEntry* __restrict__ col,
           const AxisEntry* __restrict__ rowz, const ViewEntry* __restrict__ view, DetGrid G,
           int nx, int ny, int nz, int na, int nb, int nv, float dz,
           const int* __restrict__ skip, int xfold, int w0, int w1, int first, int last,
           float2* __restrict__ dq, int dqz, int lanes)
{
    if (skip && *skip) return;
    const int lz = FULL ? 5 : lanes;
    constexpr int NI = 2 * NR, NP = PB * PB;            // images, columns of a block
    __shared__ ReflCand<NP> cand[kReflWarps][32];
    const ReflGeom g = refl_geom(NR, nv, na, nb);
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int nzw = nz / 2, hx = nx / 2, hy = ny / 2, nbh = g.nbh;
    // the lane's group of ZL = 2^lz lanes, its first lane and lanes' mask
    const int ZL = 1 << lz, g0 = FULL ? 0 : lane & ~(ZL - 1), sub = lane & (ZL - 1);
    const unsigned gm = FULL ? 0xffffffffu : (0xffffffffu >> (32 - ZL)) << g0;
    const int X0 = PB * (((2 * blockIdx.x + (wp & 1)) << (5 - lz)) + (g0 >> lz));
    const int Y0 = PB * (2 * blockIdx.y + (wp >> 1));
    const bool have = X0 < hx && Y0 < hy && !(NR == 4 && X0 > Y0);
    const unsigned wm = FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, have);
    if (!have) return;                                  // whole groups
    const int z = (blockIdx.z << lz) + sub;
    const bool on = z < nzw;
    // column c = (X0 + c % PB, Y0 + c / PB); P: the sums the turn slots feed, Q:
    // the reflected slots' (rotated one place per image, in opposite
    // directions; exchanged between the C and the D images)
    float2 P[NP][NR], Q[NP][NR];
#pragma unroll
    for (int c = 0; c < NP; c++)
#pragma unroll
        for (int j = 0; j < NR; j++) { P[c][j] = make_float2(0.0f, 0.0f); Q[c][j] = P[c][j]; }
    const long long nxy = (long long)nx * ny;
    if (!first && on) {                                 // continue the chunk before
        const float* Xf = (const float*)X;
#pragma unroll
        for (int c = 0; c < NP; c++) {
            const int ix = X0 + c % PB, iy = Y0 + c / PB;
            if (NR == 4 && ix > iy) continue;
#pragma unroll
            for (int j = 0; j < NI; j++) {
                float2 a;
                if (NR == 4 && ix == iy && j >= NR) {
                    a = dq[((long long)ix * dqz + z) * NR + (j - NR)];
                } else {
                    int qx, qy;
                    refl_column<NR>(j, ix, iy, nx, ny, qx, qy);
                    const long long q = (long long)qy * nx + qx;
                    if (xfold) a = *reinterpret_cast<const float2*>(Xf + orbit_pair(qx, qy, z, nx, ny));
                    else a = make_float2(Xf[z * nxy + q], Xf[(nz - 1 - z) * nxy + q]);
                }
                if (j < NR) P[c][j % NR] = a; else Q[c][j % NR] = a;
            }
        }
    }
    const float inv_dv = 1.0f / G.dv;
    const float fz = (float)z, fz1 = (float)(z + 1);
    for (int w = w0; w <= min(w1, g.ov); w++) {
        int vt, alim;
        long long base;
        refl_view(g, w, vt, base, alim);
        const ViewEntry ve = view[vt];
        const ColEntry* cv = col + (long long)vt * na;
        const AxisEntry* rv = held(rowz + (long long)vt * nb, wm);
        const TW* yv = yw + base;
        // the images' detector windows, image (lane mod NI) in each lane
        int alo, ahi;
        {
            int bx, by; float dmin, dmax;
            refl_corner<NR, PB>(sub % NI, X0, Y0, nx, ny, bx, by);
            column_window(G, ve.c, ve.s, (float)(bx - hx), (float)(by - hy), (float)PB, (float)PB,
                          na, alo, ahi, dmin, dmax);
            alo = min(alo, na);                         // lane numbers are added to it
            ahi = min(ahi, alim - 1);
        }
        const int maxw = __reduce_max_sync(wm, ahi - alo + 1);
        if (maxw <= 0) continue;                        // no ray of this view meets the blocks
        int lg = PB == 1 ? 2 : 3;                       // 4 .. ZL candidates per image
        while (lg < lz && (1 << lg) < maxw) lg++;
        const int W = 1 << lg;
        for (int k0 = 0; k0 < NI; k0 += ZL >> lg) {
            const int kmine = k0 + (sub >> lg);
            const int lo = __shfl_sync(gm, alo, g0 + kmine % NI);
            const int hi = __shfl_sync(gm, ahi, g0 + kmine % NI);
            const int kend = min(NI - k0, ZL >> lg);
            for (int jb = 0; jb < maxw; jb += W) {      // once, or W = ZL and one image
                const int ia = lo + jb + (sub & (W - 1));
                bool ok = kmine < NI && ia <= hi && FL_IN(ia, na);
                __syncwarp(gm);
                if (ok) {
                    int bx, by;
                    refl_corner<NR, PB>(kmine, X0, Y0, nx, ny, bx, by);
                    const ColEntry ce = cv[ia];
                    ReflCand<NP>& q = cand[wp][lane];
                    // the frame and the crossings of cone_column, for each column
                    const bool xd = x_dominant(ce.x, ce.y);
                    float bh, be;
                    make_anchor<kSegCone>(xd ? ce.x : ce.y, (xd ? bx : by) >> kSegCone,
                                          xd ? nx : ny, bh, be);
                    const float mx = __fsub_rn((float)bx, ce.x.kq);
                    const float my = __fsub_rn((float)by, ce.y.kq);
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
                        const int ix = X0 + c % PB, iy = Y0 + c / PB;
                        int qx, qy;
                        refl_column<NR>(kmine, ix, iy, nx, ny, qx, qy);
                        const bool i1 = PB == 2 && qx > bx, j1 = PB == 2 && qy > by;
                        const float xa = i1 ? tx[PB - 1] : tx[0], xb = i1 ? tx[PB] : tx[1];
                        const float ya = j1 ? ty[PB - 1] : ty[0], yb = j1 ? ty[PB] : ty[1];
                        float l = fmaxf(fminf(xa, xb), fminf(ya, yb));
                        float h = fminf(fmaxf(xa, xb), fmaxf(ya, yb));
                        // outside the octant, or the D images of the diagonal
                        if (NR == 4 && (ix > iy || (ix == iy && kmine >= NR))) { l = 1.0f; h = 0.0f; }
                        q.lh[c] = make_float2(l, h);
                        if (l < h) { lmin = fminf(lmin, l); hmax = fmaxf(hmax, h); }
                    }
                    ok = lmin < hmax;
                    // absolute parameters of the block's ends (row windows only)
                    const float r1 = __fdividef(inv_dv, __fadd_rn(bh, lmin) + ve.ac);
                    const float r2 = __fdividef(inv_dv, __fadd_rn(bh, hmax) + ve.ac);
                    const float zb = -(float)(nz / 2) * dz - ve.sz, vb = G.v0 * inv_dv;
                    q.bh = bh; q.be = be;
                    q.s1 = dz * r1; q.c1 = zb * r1 - vb - 0.02f;
                    q.s2 = dz * r2; q.c2 = zb * r2 - vb + 0.02f;
                    q.off = nbh * ia;
                }
                const unsigned mask = __ballot_sync(gm, ok) >> g0;
                __syncwarp(gm);
#pragma unroll 1
                for (int k = 0; k < kend; k++) {
                    if (k0 + k == NR && jb == 0) {      // the D images: P and Q trade roles
#pragma unroll
                        for (int c = 0; c < NP; c++)
#pragma unroll
                            for (int j = 0; j < NR; j++) {
                                const float2 t = P[c][j]; P[c][j] = Q[c][j]; Q[c][j] = t;
                            }
                    }
                    unsigned todo = (mask >> (k << lg)) & (0xffffffffu >> (32 - W));
#pragma unroll 1
                    for (; todo; todo &= todo - 1) {
                        const ReflCand<NP>& q = cand[wp][g0 + (k << lg) + __ffs(todo) - 1];
                        const float bh = q.bh, be = q.be;
                        // the walked rays descend and the rows rise: the rows
                        // that meet voxel z lie between its ends' crossings
                        const int blo = max(__float2int_ru(fmaf(fz, q.s1, q.c1)), 0);
                        const int bhi = min(__float2int_rd(fmaf(fz1, q.s2, q.c2)),
                                            on ? nbh - 1 : -1);
                        const TW* yt = yv + (long long)NI * q.off;
                        float2 lh[NP];
#pragma unroll
                        for (int c = 0; c < NP; c++) lh[c] = q.lh[c];
#pragma unroll 1
                        for (int ib = blo; ib <= bhi; ib++) {
                            if (!FL_IN(ib, nbh)) continue;
                            const AxisEntry re = rv[ib];
                            float t[NI], u[NI];
                            ld_in<TW, NI>(yt + NI * ib, t);
                            ld_in<TW, NI>(yt + g.plane + NI * ib, u);
                            const float2 az = row_planes(re, fz, fz1, bh, be);
#pragma unroll
                            for (int c = 0; c < NP; c++) {
                                const float wgt = fminf(lh[c].y, az.x) - fmaxf(lh[c].x, az.y);
                                if (wgt > 0.0f) {
                                    const float2 w2 = make_float2(wgt, wgt);
#pragma unroll
                                    for (int j = 0; j < NR; j++) {
                                        P[c][j] = __ffma2_rn(w2, make_float2(t[2 * j], t[2 * j + 1]), P[c][j]);
                                        Q[c][j] = __ffma2_rn(w2, make_float2(u[2 * j], u[2 * j + 1]), Q[c][j]);
                                    }
                                }
                            }
                        }
                    }
                    if (jb + W < maxw) continue;        // more of this image's candidates
                    // next image: P rotates back one place, Q forward one
#pragma unroll
                    for (int c = 0; c < NP; c++) {
                        const float2 a = P[c][0];
#pragma unroll
                        for (int j = 0; j + 1 < NR; j++) P[c][j] = P[c][j + 1];
                        P[c][NR - 1] = a;
                        const float2 b = Q[c][NR - 1];
#pragma unroll
                        for (int j = NR - 1; j > 0; j--) Q[c][j] = Q[c][j - 1];
                        Q[c][0] = b;
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NP; c++)                    // C sums back into P
#pragma unroll
            for (int j = 0; j < NR; j++) { const float2 t = P[c][j]; P[c][j] = Q[c][j]; Q[c][j] = t; }
    }
    if (!on) return;
    // C_j = S^j V0 holds P[j] (and, on the diagonal of NR = 4, Q[j + 1], the
    // sums of D_{j+1} = C_j; before the last chunk they stay apart, Q in dq);
    // D_j = S^j M V0 holds Q[j]
#pragma unroll
    for (int c = 0; c < NP; c++) {
        const int ix = X0 + c % PB, iy = Y0 + c / PB;
        if (NR == 4 && ix > iy) continue;
        const bool diag = NR == 4 && ix == iy;
#pragma unroll
        for (int j = 0; j < NI; j++) {
            if (diag && j >= NR) {
                if (!last) dq[((long long)ix * dqz + z) * NR + (j - NR)] = Q[c][j % NR];
                continue;
            }
            float2 a = j < NR ? P[c][j % NR] : Q[c][j % NR];
            if (j < NR && diag && last) {
                const float2 b = Q[c][(j + 1) % NR];
                a.x += b.x; a.y += b.y;
            }
            int qx, qy;
            refl_column<NR>(j, ix, iy, nx, ny, qx, qy);
            if (xfold) {                                // the folded volume's orbits
                Store<TX>::st2(X + orbit_pair(qx, qy, z, nx, ny), a.x, a.y);
            } else {
                const long long q = (long long)qy * nx + qx;
                Store<TX>::st(X + z * nxy + q, a.x);
                Store<TX>::st(X + (nz - 1 - z) * nxy + q, a.y);
            }
        }
    }
}

// Warps with blocks of PB x PB columns and 2^lz lanes per block.
long long warp_count(const fl_plan* p, int PB, int lz)
{
    const fl_scan& s = p->s;
    const long long bx = fl_div_up(s.nx / 2, PB), by = fl_div_up(s.ny / 2, PB);
    const long long blocks = fl_plan_refl(p) == 4 ? bx * (bx + 1) / 2 : bx * by;
    return (blocks * fl_div_up(s.nz / 2, 1 << lz)) >> (5 - lz);
}

int lanes_log2(const fl_plan* p, int PB)
{
    return adj_lanes_log2(p, p->s.nz / 2, 3, [&](int lz) { return warp_count(p, PB, lz); });
}

template <typename TX, typename TW>
void launch(fl_plan* p, const void* yw, void* x, const int* skip, int xfold, cudaStream_t st)
{
    const fl_scan& s = p->s;
    const int NR = fl_plan_refl(p), nzw = s.nz / 2;
    const int PB = fl_plan_adj_run(p), lz = lanes_log2(p, PB);
    const dim3 grid(fl_div_up(s.nx / 2, (2 * PB) << (5 - lz)), fl_div_up(s.ny / 2, 2 * PB),
                    fl_div_up(nzw, 1 << lz));
    // view chunks (fl_plan_adj_chunks): launches over consecutive walked
    // views, so the blocks resident together read the same views' rows from
    // L2; FP32 output only
    const int nch = fl_plan_adj_chunks(p, std::is_same<TX, float>::value);
    const int wper = (refl_geom(NR, s.nv, s.na, s.nb).ov + nch) / nch;
    auto* k = k_adj_refl<TX, 2, TW, 4, true>;
#define FL_PICK(PB_, NR_) \
    if (PB == PB_ && NR == NR_) \
        k = lz == 5 ? k_adj_refl<TX, PB_, TW, NR_, true> : k_adj_refl<TX, PB_, TW, NR_, false>
    FL_PICK(2, 4);
    FL_PICK(1, 4);
    FL_PICK(2, 2);
    FL_PICK(1, 2);
#undef FL_PICK
    for (int c = 0; c < nch; c++)
        k<<<grid, kReflWarps * 32, 0, st>>>((TX*)x, (const TW*)yw, p->d_col, p->d_rowz, p->d_view,
                                            det_grid(p), s.nx, s.ny, s.nz, s.na, s.nb, s.nv, s.dz,
                                            skip, xfold, c * wper, c * wper + wper - 1, c == 0,
                                            c == nch - 1, p->d_dq, nzw, lz);
}

}  // namespace

// 2 x 2 columns per warp load a row's orbit once for all of them, but make a
// quarter of the warps: they pay once those fill the GPU (160^3, 200 views:
// 1.46 ms against 1.59 with one column; 128^3, 120 views, 1,056 warps: 0.74
// against 0.49). A warp takes three times as long, so not where more of its lanes
// have no voxel than one column's would (256 x 256 x 24, 360 views: 1.00 ms with 32
// lanes, 0.71 with 16 and one column).
int fl_plan_adj_run(const fl_plan* p)
{
    if (p->adj_run) return p->adj_run;
    const long long w2 = warp_count(p, 2, lanes_log2(p, 2)), w1 = warp_count(p, 1, lanes_log2(p, 1));
    return w2 >= adj_full_warps(p) && 3 * w2 < w1 ? 2 : 1;
}

void fl_matched_adjoint_refl(fl_plan* p, const void* yw, int wt, void* x, int xt, const int* skip,
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

FL_OOB_ACCESSOR(fl_oob_refl)
