// framelet.cu -- undecimated tensor-product framelets (Haar, piecewise linear,
// piecewise cubic), soft-shrinkage and the fused split-Bregman update.
//
// Semantics (FraDecMultiLevel3D.m:14-47, FraRecMultiLevel3D.m:14-48,
// ConvSymAsym3D.m:18-34, GenerateFrameletFilter.m:2-30, softThreshold.m:47-80):
//  * every 1-D filter is a circular correlation, taps at offsets
//    (t - c) * 2^(level-1) around the output sample (imfilter 'circular');
//  * 3-D band (i, j, k): D_i along y, D_j along x, D_k along z; 2-D band
//    (i, j): D_i along x, D_j along y (FraDecMultiLevel2D.m:43-52);
//  * level l+1 decomposes the low band (0,0[,0]) of level l; the synthesis
//    replaces that low band by the reconstruction of level l+1, so the low
//    band of every level but the last is never stored here;
//  * soft-shrink sign(a) max(|a| - tau, 0) applies to every stored band except
//    the low band of the last level.
// Coefficient layout: level-major; inside a level, band index = base-nf digits
// in pass order (nf filters per axis; linear 3-D: 9i + 3j + k, 2-D: 3i + j),
// band 0 omitted below the last level; each band is one volume (x fastest).
//
// Every pass is a streaming circular stencil along one axis. The last analysis
// pass computes each band value in registers and applies the Bregman update
// (v, alpha, alpha - v) without storing W u; the last synthesis pass writes
// b = base + mu * W^T t directly.
#include <cstring>
#include <new>
#include <vector>

#include "fl_trace.h"
#include "fl_common.cuh"

namespace {

constexpr int kMaxBands = 125;   // cubic bank in 3-D: 5^3 bands

struct Filters {
    float f[5][5];   // up to 5 filters x 5 taps (linear 3 x 3, haar 2 x 3, cubic 5 x 5)
    int nf, nt;      // filters, taps
};

struct BandPtrs {
    float* p[kMaxBands];   // per band: coefficient array (nullptr: not stored)
};

// j mod n for a tap index; |j - [0, n)| is almost always below n, so one add
// or subtract wraps it (the modulo only runs for volumes smaller than a tap
// offset)
__device__ __forceinline__ int wrapi(int j, int n)
{
    if (j < 0) {
        j += n;
        if (j < 0) { j %= n; if (j < 0) j += n; }
    } else if (j >= n) {
        j -= n;
        if (j >= n) j %= n;
    }
    return j;
}

// index of the neighbour at offset d along AXIS (0 x, 1 y, 2 z), circular
template <int AXIS>
__device__ __forceinline__ long long nb(int ix, int iy, int iz, int nx, int ny, int nz, int d)
{
    if (AXIS == 0) ix = wrapi(ix + d, nx);
    else if (AXIS == 1) iy = wrapi(iy + d, ny);
    else iz = wrapi(iz + d, nz);
    return ((long long)iz * ny + iy) * nx + ix;
}

// Every pass runs on the grid (x in blocks of 128, y, z * channel): no index
// arithmetic per element beyond the wrap of the taps. NF filters of NT taps.
constexpr int kPassThreads = 128;

// out[NF*c + f] = F_f (*) in[c] along AXIS   (analysis split pass)
template <int NF, int NT, int AXIS>
__global__ void __launch_bounds__(kPassThreads)
k_split(const float* __restrict__ in, long long in_stride, float* __restrict__ out,
        long long out_stride, int nx, int ny, int nz, int step, Filters F)
{
    const int ix = blockIdx.x * kPassThreads + threadIdx.x;
    if (ix >= nx) return;
    const int iy = blockIdx.y, iz = blockIdx.z % nz, c = blockIdx.z / nz;
    const long long q = ((long long)iz * ny + iy) * nx + ix;
    const float* src = in + (long long)c * in_stride;
    constexpr int ctr = (NT - 1) / 2;
    float v[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) v[t] = __ldg(src + nb<AXIS>(ix, iy, iz, nx, ny, nz, (t - ctr) * step));
#pragma unroll
    for (int f = 0; f < NF; f++) {
        float s = 0.0f;
#pragma unroll
        for (int t = 0; t < NT; t++) s = fmaf(F.f[f][t], v[t], s);
        out[(long long)(NF * c + f) * out_stride + q] = s;
    }
}

// Last analysis pass. band = NF*c + f. mode 0: coef[band] = w (skipping band 0
// below the last level, which goes to `low`); mode 1: split-Bregman update on
// v and t = alpha - v_new with soft threshold tau (no shrink on band 0 of the
// last level).
template <int NF, int NT, int AXIS>
__global__ void __launch_bounds__(kPassThreads)
k_split_last(const float* __restrict__ in, long long in_stride, int nx, int ny, int nz,
             int step, Filters F, BandPtrs coef, BandPtrs tout, float* __restrict__ low,
             int last, int mode, float tau)
{
    const int ix = blockIdx.x * kPassThreads + threadIdx.x;
    if (ix >= nx) return;
    const int iy = blockIdx.y, iz = blockIdx.z % nz, c = blockIdx.z / nz;
    const long long q = ((long long)iz * ny + iy) * nx + ix;
    const float* src = in + (long long)c * in_stride;
    constexpr int ctr = (NT - 1) / 2;
    float v[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) v[t] = __ldg(src + nb<AXIS>(ix, iy, iz, nx, ny, nz, (t - ctr) * step));
    float vv[NF];                                          // v of every band, read before any store
#pragma unroll
    for (int f = 0; f < NF; f++)
        vv[f] = (mode == 0 || (NF * c + f == 0 && !last)) ? 0.0f : coef.p[NF * c + f][q];
#pragma unroll
    for (int f = 0; f < NF; f++) {
        float w = 0.0f;
#pragma unroll
        for (int t = 0; t < NT; t++) w = fmaf(F.f[f][t], v[t], w);
        const int band = NF * c + f;
        if (band == 0 && !last) {
            if (low) low[q] = w;
            continue;
        }
        if (mode == 0) {
            coef.p[band][q] = w;
        } else {
            const float s = vv[f] + w;                     // v + W u
            float a = s;                                   // alpha
            if (!(band == 0 && last)) {
                const float m = fabsf(s) - tau;
                a = m > 0.0f ? copysignf(m, s) : 0.0f;
            }
            const float vn = s - a;                        // v + W u - alpha
            coef.p[band][q] = vn;
            tout.p[band][q] = a - vn;                      // alpha - v_new
        }
    }
}

// out[c] = sum_f F_f (*) in[NF*c + f] along AXIS (synthesis merge pass); input
// arrays come from `bands` (band pointer per index) -- with band 0 replaced by
// `low` when non-null. final: out = base + scale * result.
template <int NF, int NT, int AXIS>
__global__ void __launch_bounds__(kPassThreads)
k_merge(BandPtrs bands, const float* __restrict__ low, float* __restrict__ out,
        long long out_stride, int nx, int ny, int nz, int step, Filters F,
        const float* __restrict__ base, float scale, int final_)
{
    const int ix = blockIdx.x * kPassThreads + threadIdx.x;
    if (ix >= nx) return;
    const int iy = blockIdx.y, iz = blockIdx.z % nz, c = blockIdx.z / nz;
    const long long q = ((long long)iz * ny + iy) * nx + ix;
    constexpr int ctr = (NT - 1) / 2;
    float s = 0.0f;
#pragma unroll
    for (int f = 0; f < NF; f++) {
        const int band = NF * c + f;
        const float* src = (band == 0 && low) ? low : bands.p[band];
#pragma unroll
        for (int t = 0; t < NT; t++)
            s = fmaf(F.f[f][t], __ldg(src + nb<AXIS>(ix, iy, iz, nx, ny, nz, (t - ctr) * step)), s);
    }
    if (final_) s = (base ? __ldg(base + q) : 0.0f) + scale * s;
    out[(long long)c * out_stride + q] = s;
}

// launchers: filter bank (NF, NT) and axis as template arguments
template <int NF, int NT>
struct Pass {
    static void split(int axis, dim3 g, cudaStream_t s, const float* in, long long is, float* out,
                      long long os, int nx, int ny, int nz, int step, const Filters& F)
    {
        if (axis == 0) k_split<NF, NT, 0><<<g, kPassThreads, 0, s>>>(in, is, out, os, nx, ny, nz, step, F);
        else if (axis == 1) k_split<NF, NT, 1><<<g, kPassThreads, 0, s>>>(in, is, out, os, nx, ny, nz, step, F);
        else k_split<NF, NT, 2><<<g, kPassThreads, 0, s>>>(in, is, out, os, nx, ny, nz, step, F);
    }
    static void split_last(int axis, dim3 g, cudaStream_t s, const float* in, long long is,
                           int nx, int ny, int nz, int step, const Filters& F, const BandPtrs& cb,
                           const BandPtrs& tb, float* low, int last, int mode, float tau)
    {
        if (axis == 0)
            k_split_last<NF, NT, 0><<<g, kPassThreads, 0, s>>>(in, is, nx, ny, nz, step, F, cb, tb, low, last, mode, tau);
        else if (axis == 1)
            k_split_last<NF, NT, 1><<<g, kPassThreads, 0, s>>>(in, is, nx, ny, nz, step, F, cb, tb, low, last, mode, tau);
        else
            k_split_last<NF, NT, 2><<<g, kPassThreads, 0, s>>>(in, is, nx, ny, nz, step, F, cb, tb, low, last, mode, tau);
    }
    static void merge(int axis, dim3 g, cudaStream_t s, const BandPtrs& b, const float* low,
                      float* out, long long os, int nx, int ny, int nz, int step,
                      const Filters& F, const float* base, float scale, int final_)
    {
        if (axis == 0)
            k_merge<NF, NT, 0><<<g, kPassThreads, 0, s>>>(b, low, out, os, nx, ny, nz, step, F, base, scale, final_);
        else if (axis == 1)
            k_merge<NF, NT, 1><<<g, kPassThreads, 0, s>>>(b, low, out, os, nx, ny, nz, step, F, base, scale, final_);
        else
            k_merge<NF, NT, 2><<<g, kPassThreads, 0, s>>>(b, low, out, os, nx, ny, nz, step, F, base, scale, final_);
    }
};

// ---------------------------------------------------------------------------
// z-streaming 3-D level kernels for the three-tap banks (linear, Haar). A
// block owns a column tile (warp = one row y, lane = x) and walks the slices
// z = r, r + s, r + 2s, ... of one residue class r mod s (s = 2^level), up to
// seg_len output slices. The z taps of an output slice are the slices z - s, z,
// z + s of its own class, so each thread keeps the z-pass inputs of its
// sample in a three-slot register window and every slice is read once per
// block. Every value is the same fmaf chain as in the separable pass kernels
// above (taps in order, filters in order), so both forms give identical bits.
constexpr int kSX = 32, kSY = 8, kST = kSX * kSY;   // column tile, threads per block
constexpr int kRowMax = 512;                         // k_syn_zx: longest whole row
constexpr int kMaxStreamStep = 8;                    // dilations the streaming kernels take

// element of a plane: a base that all threads share and a 32-bit byte offset,
// which the load and store instructions add themselves
template <typename T>
__device__ __forceinline__ T* at(T* plane, unsigned off)
{
    return (T*)((const char*)plane + off);
}

// slices of residue class r in [0, nz): r, r + s, ...
__host__ __device__ inline int class_len(int nz, int s, int r)
{
    return r < nz ? (nz - 1 - r) / s + 1 : 0;
}

// resident blocks of k_ana_stream per SM: three, and two where 27 values of v
// are held as well as the window
__host__ __device__ constexpr int ana_resident(int nf, int mode) { return nf == 3 && mode == 1 ? 2 : 3; }

// resident threads of k_syn_zx per SM. Four bands a thread (Haar) leave too few loads
// in flight with two blocks of 512: 200^3, one level 114 us with 1024 threads, 98
// with 1536 (a slice more ahead 107, two 101); 256^3 193 and 170.
__host__ __device__ constexpr int syn_threads(int nf) { return nf == 2 ? 1536 : 1024; }

// One analysis level: the y and x passes of each slice in shared memory, the
// z pass from the register window, fused with the coefficient write (MODE 0)
// or the Bregman update (MODE 1) exactly as k_split_last. The stores of 27
// arrays bound it. MODE 0 needs 72 registers, so three blocks fit; the window
// is used by turns (no moves), a store adds a 32-bit offset to its band's plane,
// and the x pass reads its own warp's row only, so one barrier a slice is left:
// 256^3, two levels, linear bank 692 -> 624 us (5.9 of 6.7 TB/s). MODE 1 reads
// all v of the next output before the slice's barrier, ahead of every store
// (the band pointers may alias as far as the compiler knows): with the
// synthesis 2757 -> 2530 us; v by groups of channels, as few as three in flight
// beside as many in use, gave 2570-3290 us, also with three blocks.
template <int NF, int S, int MODE>
__global__ void __launch_bounds__(kST, ana_resident(NF, MODE))
k_ana_stream(const float* __restrict__ in, int nx, int ny, int nz, int nseg, int seg_len, Filters F,
             BandPtrs coef, BandPtrs tout, float* __restrict__ low, int last, float tau)
{
    constexpr int RX = kSX + 2 * S, RY = kSY + 2 * S;   // in-plane region (halo S)
    constexpr int XR = RX - 32;                        // lanes holding a second column
    constexpr int LR = (RY + kSY - 1) / kSY;           // region rows per warp
    constexpr int NC = NF * NF;                        // channels into the z pass
    __shared__ float s_in[2][RY][RX];
    __shared__ float s_p1[NF][kSY][RX];               // a warp writes and reads only its own row
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int x0 = blockIdx.x * kSX, y0 = blockIdx.y * kSY;
    const int seg = blockIdx.z % nseg, r = blockIdx.z / nseg;
    const int nfirst = seg * seg_len, nend = min(nfirst + seg_len, class_len(nz, S, r));
    if (nfirst >= nend) return;                        // uniform per block
    const int xa = wrapi(x0 - S + lane, nx);
    const int xb = lane < XR ? wrapi(x0 - S + 32 + lane, nx) : 0;
    int rows[LR];
#pragma unroll
    for (int m = 0; m < LR; m++) rows[m] = wrapi(y0 - S + wy + kSY * m, ny);
    const int x = x0 + lane, y = y0 + wy;
    const bool ok = x < nx && y < ny;
    float pa[LR], pb[LR];                              // the next slice's region, in flight
    auto fetch = [&](int n) {
        const long long zo = (long long)wrapi(r + S * n, nz) * ny;
#pragma unroll
        for (int m = 0; m < LR; m++)
            if (wy + kSY * m < RY) {
                const float* row = in + (zo + rows[m]) * nx;
                pa[m] = __ldg(row + xa);
                pb[m] = lane < XR ? __ldg(row + xb) : 0.0f;
            }
    };
    const long long plane = (long long)ny * nx;
    const unsigned off = 4u * ((unsigned)y * nx + x);
    float vv[MODE ? NC * NF : 1];                      // mode 1: v of the next output
    float win[3][NC];                                  // the slices z - S, z, z + S by turns
    fetch(nfirst - 1);
    for (int n = nfirst - 1, b = 0;;) {
#pragma unroll
        for (int u = 0; u < 3; u++, n++, b ^= 1) {
            if (n > nend) return;                      // uniform per block
#pragma unroll
            for (int m = 0; m < LR; m++)
                if (wy + kSY * m < RY) {
                    s_in[b][wy + kSY * m][lane] = pa[m];
                    if (lane < XR) s_in[b][wy + kSY * m][32 + lane] = pb[m];
                }
            if (n < nend) fetch(n + 1);
            const long long zo = (r + S * (n - 1)) * plane;   // slots: z - S, z, z + S
            if (MODE == 1 && n > nfirst && ok) {
#pragma unroll
                for (int band = 0; band < NC * NF; band++)
                    if (band || last) vv[band] = *at(coef.p[band] + zo, off);
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < NF; i++) {             // y pass (D_i)
                float s0 = 0.0f;
#pragma unroll
                for (int t = 0; t < 3; t++) s0 = fmaf(F.f[i][t], s_in[b][wy + t * S][lane], s0);
                s_p1[i][wy][lane] = s0;
                if (lane < XR) {
                    float s1 = 0.0f;
#pragma unroll
                    for (int t = 0; t < 3; t++) s1 = fmaf(F.f[i][t], s_in[b][wy + t * S][32 + lane], s1);
                    s_p1[i][wy][32 + lane] = s1;
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < NF; i++)               // x pass (D_j) into the newest slot
#pragma unroll
                for (int j = 0; j < NF; j++) {
                    float s0 = 0.0f;
#pragma unroll
                    for (int t = 0; t < 3; t++) s0 = fmaf(F.f[j][t], s_p1[i][wy][lane + t * S], s0);
                    win[u][NF * i + j] = s0;
                }
            if (n < nfirst + 1 || !ok) continue;       // window filling, or outside the volume
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int k = 0; k < NF; k++) {         // z pass (D_k)
                    const int band = NF * c + k;
                    float w = 0.0f;
#pragma unroll
                    for (int t = 0; t < 3; t++) w = fmaf(F.f[k][t], win[(u + 1 + t) % 3][c], w);
                    if (band == 0 && !last) {
                        if (low) *at(low + zo, off) = w;
                        continue;
                    }
                    if (MODE == 0) {
                        *at(coef.p[band] + zo, off) = w;
                    } else {
                        const float sv = vv[band] + w; // v + W u
                        float a = sv;                  // alpha
                        if (!(band == 0 && last)) {
                            const float mg = fabsf(sv) - tau;
                            a = mg > 0.0f ? copysignf(mg, sv) : 0.0f;
                        }
                        const float vn = sv - a;       // v + W u - alpha
                        *at(coef.p[band] + zo, off) = vn;
                        *at(tout.p[band] + zo, off) = a - vn;   // alpha - v_new
                    }
                }
        }
    }
}

// The z and x merges of one synthesis level (k_merge along z into NF^2
// arrays, then along x into the NF arrays A_i), band 0 taken from `low` when
// non-null. Threads along x hold aligned runs of columns: a whole row where it
// fits in kRowMax threads (`whole`, several rows a block when it is short),
// else a tile of them and one warp more for the columns beside it. The x
// taps come from shared memory. blockIdx.z = seg + nseg (i + NF r).
// The 27 bands' reads bound it; issue slots came next. Warps of 32 - 2S outputs
// whose taps came by shuffles read rows from unaligned columns, and moving the
// window and adding 64-bit addresses took half of the 135 instructions a
// slice: 256^3, two levels, with the y merge 916 -> 759 us. Copies into a ring in
// shared memory, four slices deep, were slower (968 us).
template <int NF, int S>
__global__ void __launch_bounds__(kRowMax, syn_threads(NF) / kRowMax)
k_syn_zx(BandPtrs bands, const float* __restrict__ low, float* __restrict__ A, long long N,
         int nx, int ny, int nz, int nseg, int seg_len, int whole, Filters R)
{
    constexpr int NB = NF * NF;                        // bands per thread
    extern __shared__ float s_bm[];                    // [2][NF][rows][blockDim.x]
    const int W = blockDim.x, rows = blockDim.y, tx = threadIdx.x, T = W - 32;
    const int y = blockIdx.y * rows + threadIdx.y;
    const int seg = blockIdx.z % nseg, ir = blockIdx.z / nseg, i = ir % NF, r = ir / NF;
    const int nfirst = seg * seg_len, nend = min(nfirst + seg_len, class_len(nz, S, r));
    if (nfirst >= nend) return;                        // uniform per block
    // this thread's column and the places of its x neighbours in its row
    int x, left, right;
    bool out_ok = y < ny;
    if (whole) {
        x = min(tx, nx - 1);
        left = wrapi(x - S, nx);
        right = wrapi(x + S, nx);
        out_ok = out_ok && tx < nx;
    } else {
        // the last warp holds the S columns before the tile, then the S after it
        const int x0 = blockIdx.x * T, h = tx - T;
        const int off = h < 0 ? tx : h < S ? h - S : min(h - S, S - 1) + T;
        x = wrapi(x0 + off, nx);
        left = h < 0 ? (tx < S ? T + tx : tx - S) : tx;
        right = h < 0 ? (tx + S < T ? tx + S : tx + S + S) : tx;
        out_ok = out_ok && h < 0 && x0 + off < nx;
    }
    const long long plane = (long long)ny * nx;
    const unsigned off = 4u * ((unsigned)min(y, ny - 1) * nx + x);
    auto src = [&](int b) -> const float* {            // b = NF j + k: band NF (NF i + j) + k
        const int band = NF * NF * i + b;
        return (band == 0 && low) ? low : bands.p[band];
    };
    const int row = threadIdx.y * W, step = rows * W;
    float w[4][NB];                                    // three taps and the next slice, by turns
    auto fetch = [&](int n, float (&d)[NB]) {
        const long long zo = wrapi(r + S * n, nz) * plane;
#pragma unroll
        for (int b = 0; b < NB; b++) d[b] = __ldg(at(src(b) + zo, off));
    };
    fetch(nfirst - 1, w[0]);
    fetch(nfirst, w[1]);
    fetch(nfirst + 1, w[2]);
    for (int n = nfirst + 1;;) {
#pragma unroll
        for (int u = 0; u < 4; u++, n++) {
            if (n > nend) return;                      // uniform per block
            if (n < nend) fetch(n + 1, w[(u + 3) & 3]);
            float* bm = s_bm + (u & 1) * NF * step + row;   // double-buffered: one barrier a slice
            float own[NF];
#pragma unroll
            for (int j = 0; j < NF; j++) {
                float m = 0.0f;                        // z merge (R_k) of channel NF i + j
#pragma unroll
                for (int k = 0; k < NF; k++)
#pragma unroll
                    for (int t = 0; t < 3; t++) m = fmaf(R.f[k][t], w[(u + t) & 3][NF * j + k], m);
                own[j] = m;
                bm[j * step + tx] = m;
            }
            __syncthreads();
            float a = 0.0f;                            // output slice r + S (n - 1)
#pragma unroll
            for (int j = 0; j < NF; j++) {             // x merge (R_j)
                a = fmaf(R.f[j][0], bm[j * step + left], a);
                a = fmaf(R.f[j][1], own[j], a);
                a = fmaf(R.f[j][2], bm[j * step + right], a);
            }
            if (out_ok) *at(A + i * N + (r + S * (n - 1)) * plane, off) = a;
        }
    }
}

// The y merge of one synthesis level (k_merge along y into the output, final
// = base + scale * result), streaming along y: a thread owns one column
// (x, z) and walks the rows of one residue class mod S, the three y taps of
// each output row held in a register window per input array.
constexpr int kSegY = 8;                             // output rows of one class per thread: 32 left
                                                     // too few threads (77 x 61 x 45: 69 -> 44 us)

template <int NF, int S>
__global__ void __launch_bounds__(128)
k_merge_y_stream(const float* __restrict__ A, long long N, float* __restrict__ out, int nx,
                 int ny, int nz, int nseg, Filters R, const float* __restrict__ base,
                 float scale, int final_)
{
    const int x = blockIdx.x * 128 + threadIdx.x, z = blockIdx.y;
    const int seg = blockIdx.z % nseg, r = blockIdx.z / nseg;
    const int nfirst = seg * kSegY, nend = min(nfirst + kSegY, class_len(ny, S, r));
    if (x >= nx || nfirst >= nend) return;
    const long long zo = (long long)z * ny * nx + x;
    float win[3][NF], nxt[NF];
    auto fetch = [&](int n, float (&d)[NF]) {
        const long long o = zo + (long long)wrapi(r + S * n, ny) * nx;
#pragma unroll
        for (int i = 0; i < NF; i++) d[i] = __ldg(A + i * N + o);
    };
    fetch(nfirst - 1, win[1]);
    fetch(nfirst, win[2]);
    fetch(nfirst + 1, nxt);
    for (int n = nfirst + 1; n <= nend; n++) {
#pragma unroll
        for (int i = 0; i < NF; i++) { win[0][i] = win[1][i]; win[1][i] = win[2][i]; win[2][i] = nxt[i]; }
        if (n < nend) fetch(n + 1, nxt);
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < NF; i++)
#pragma unroll
            for (int t = 0; t < 3; t++) sum = fmaf(R.f[i][t], win[t][i], sum);
        const long long q = zo + (long long)(r + S * (n - 1)) * nx;
        if (final_) sum = (base ? __ldg(base + q) : 0.0f) + scale * sum;
        out[q] = sum;
    }
}

unsigned grid_for(long long n)
{
    long long g = (n + 255) / 256;
    return (unsigned)(g < 4096 ? (g > 0 ? g : 1) : 4096);
}

}  // namespace

// ---------------------------------------------------------------------------
// out = sign(a) max(|a| - tau, 0) for coefficients outside [keep0, keep1)
// (the unshrunk low band), out = a inside
__global__ void k_shrink(const float* __restrict__ a, float* __restrict__ out, long long n,
                         long long keep0, long long keep1, float tau)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float v = a[i];
        if (i >= keep0 && i < keep1) { out[i] = v; continue; }
        const float m = fmaxf(fabsf(v) - tau, 0.0f);
        out[i] = v > 0.0f ? m : (v < 0.0f ? -m : 0.0f);
    }
}

struct fl_framelet {
    int nx, ny, nz, dim, levels, kind;
    int nf, nbands;                 // filters per axis, bands per level (nf^dim)
    long long N;
    Filters D, R;
    int axes[3];                    // analysis pass order
    int fused;                      // 3-D levels through the z-streaming kernels
    int sms;                        // multiprocessors of the device
    float* work;                    // intermediates: nf^(dim-1) + nf^(dim-2) arrays + low
    long long work_elems;
    std::vector<long long> level_base;   // first coefficient band of each level
    long long ncoef_bands;
};

static void set_filters(fl_framelet* w, int kind)
{
    std::memset(&w->D, 0, sizeof w->D);
    std::memset(&w->R, 0, sizeof w->R);
    const float r2 = 1.41421356237309505f;
    if (kind == 1) {   // piecewise linear (GenerateFrameletFilter.m:9-17)
        const float d[3][3] = {{0.25f, 0.5f, 0.25f}, {-r2 / 4, 0.0f, r2 / 4}, {-0.25f, 0.5f, -0.25f}};
        const float r[3][3] = {{0.25f, 0.5f, 0.25f}, {r2 / 4, 0.0f, -r2 / 4}, {-0.25f, 0.5f, -0.25f}};
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) { w->D.f[a][b] = d[a][b]; w->R.f[a][b] = r[a][b]; }
        w->D.nf = w->R.nf = 3; w->D.nt = w->R.nt = 3;
    } else if (kind == 3) {   // piecewise cubic (GenerateFrameletFilter.m:18-30)
        const float r6 = 2.44948974278317810f;
        const float d[5][5] = {{1 / 16.f, 4 / 16.f, 6 / 16.f, 4 / 16.f, 1 / 16.f},
                               {-1 / 8.f, -2 / 8.f, 0.f, 2 / 8.f, 1 / 8.f},
                               {-r6 / 16, 0.f, 2 * r6 / 16, 0.f, -r6 / 16},
                               {-1 / 8.f, 2 / 8.f, 0.f, -2 / 8.f, 1 / 8.f},
                               {-1 / 16.f, 4 / 16.f, -6 / 16.f, 4 / 16.f, -1 / 16.f}};
        const float r[5][5] = {{1 / 16.f, 4 / 16.f, 6 / 16.f, 4 / 16.f, 1 / 16.f},
                               {1 / 8.f, 2 / 8.f, 0.f, -2 / 8.f, -1 / 8.f},
                               {-r6 / 16, 0.f, 2 * r6 / 16, 0.f, -r6 / 16},
                               {1 / 8.f, -2 / 8.f, 0.f, 2 / 8.f, -1 / 8.f},
                               {-1 / 16.f, 4 / 16.f, -6 / 16.f, 4 / 16.f, -1 / 16.f}};
        for (int a = 0; a < 5; a++)
            for (int b = 0; b < 5; b++) { w->D.f[a][b] = d[a][b]; w->R.f[a][b] = r[a][b]; }
        w->D.nf = w->R.nf = 5; w->D.nt = w->R.nt = 5;
    } else {           // Haar (GenerateFrameletFilter.m:2-8)
        const float d[2][3] = {{0.0f, 0.5f, 0.5f}, {0.0f, -0.5f, 0.5f}};
        const float r[2][3] = {{0.5f, 0.5f, 0.0f}, {0.5f, -0.5f, 0.0f}};
        for (int a = 0; a < 2; a++)
            for (int b = 0; b < 3; b++) { w->D.f[a][b] = d[a][b]; w->R.f[a][b] = r[a][b]; }
        w->D.nf = w->R.nf = 2; w->D.nt = w->R.nt = 3;
    }
}

extern "C" int fl_framelet_create(int nx, int ny, int nz, int levels, int kind, fl_framelet** out)
{
    FL_RANGE("fl_framelet_create");
    if (!out || nx < 1 || ny < 1 || nz < 1 || levels < 1 || levels > 8)
        return fl_set_error(FL_ERR_INVALID, "fl_framelet_create: bad size or levels");
    if (kind != FL_FRAMELET_LINEAR && kind != FL_FRAMELET_HAAR && kind != FL_FRAMELET_CUBIC)
        return fl_set_error(FL_ERR_INVALID, "fl_framelet_create: unknown filter bank %d", kind);
    {   // the passes run on the grid (x blocks, y, z * channels)
        const long long maxch = (kind == FL_FRAMELET_CUBIC ? 25 : 9);
        if (ny > 65535 || (long long)nz * maxch > 65535)
            return fl_set_error(FL_ERR_UNSUPPORTED,
                                "fl_framelet_create: ny must be <= 65535 and nz <= %lld",
                                65535 / maxch);
    }
    *out = nullptr;
    fl_framelet* w = new (std::nothrow) fl_framelet;
    if (!w) return fl_set_error(FL_ERR_ALLOC, "out of host memory");
    w->nx = nx; w->ny = ny; w->nz = nz; w->dim = (nz > 1) ? 3 : 2; w->levels = levels;
    w->kind = kind; w->N = (long long)nx * ny * nz; w->fused = 1;
    set_filters(w, kind);
    w->nf = w->D.nf;
    w->nbands = w->dim == 3 ? w->nf * w->nf * w->nf : w->nf * w->nf;
    if (w->dim == 3) { w->axes[0] = 1; w->axes[1] = 0; w->axes[2] = 2; }   // y, x, z
    else { w->axes[0] = 0; w->axes[1] = 1; w->axes[2] = -1; }              // x, y
    long long b = 0;
    for (int l = 0; l < levels; l++) {
        w->level_base.push_back(b);
        b += (l == levels - 1) ? w->nbands : w->nbands - 1;
    }
    w->ncoef_bands = b;
    long long inter = (w->dim == 3) ? (w->nf + w->nf * w->nf) : w->nf;
    w->work_elems = (inter + 2) * w->N;   // pass intermediates + two low-band volumes
    int st = fl_check_cuda(fl_malloc((void**)&w->work, w->work_elems * sizeof(float)),
                           "fl_malloc(framelet)");
    if (st) { delete w; return st; }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&w->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || w->sms < 1)
        w->sms = 152;
    *out = w;
    return fl_set_error(FL_OK, "");
}

extern "C" void fl_framelet_destroy(fl_framelet* w)
{
    if (!w) return;
    if (w->work) cudaFree(w->work);
    delete w;
}

extern "C" int64_t fl_framelet_ncoef(const fl_framelet* w)
{
    return w ? w->ncoef_bands * w->N : 0;
}

// band pointers of one level inside a coefficient set (band 0 below the last
// level is absent)
static BandPtrs level_bands(const fl_framelet* w, float* coef, int l)
{
    BandPtrs B;
    for (int b = 0; b < kMaxBands; b++) B.p[b] = nullptr;
    if (!coef) return B;
    const bool last = (l == w->levels - 1);
    long long base = w->level_base[l];
    for (int b = 0; b < w->nbands; b++) {
        if (b == 0 && !last) continue;
        long long idx = base + (last ? b : b - 1);
        B.p[b] = coef + idx * w->N;
    }
    return B;
}

static dim3 pass_grid(const fl_framelet* w, int channels)
{
    return dim3(fl_div_up(w->nx, kPassThreads), w->ny, (unsigned)(w->nz * channels));
}

// One analysis level: the separable passes along the three (two) axes, the
// last one fused with the coefficient write or the Bregman update.
template <int NF, int NT>
static void analysis_level(fl_framelet* w, const float* in, int step, const BandPtrs& cb,
                           const BandPtrs& tb, float* low_out, int last, int mode, float tau,
                           cudaStream_t s)
{
    using P = Pass<NF, NT>;
    const long long N = w->N;
    float* A = w->work;                          // NF arrays
    float* Bm = A + (long long)NF * N;           // NF^2 arrays (3-D)
    if (w->dim == 3) {
        P::split(w->axes[0], pass_grid(w, 1), s, in, N, A, N, w->nx, w->ny, w->nz, step, w->D);
        P::split(w->axes[1], pass_grid(w, NF), s, A, N, Bm, N, w->nx, w->ny, w->nz, step, w->D);
        P::split_last(w->axes[2], pass_grid(w, NF * NF), s, Bm, N, w->nx, w->ny, w->nz, step,
                      w->D, cb, tb, low_out, last, mode, tau);
    } else {
        P::split(w->axes[0], pass_grid(w, 1), s, in, N, A, N, w->nx, w->ny, w->nz, step, w->D);
        P::split_last(w->axes[1], pass_grid(w, NF), s, A, N, w->nx, w->ny, w->nz, step, w->D,
                      cb, tb, low_out, last, mode, tau);
    }
}

// One synthesis level: the merge passes in reverse axis order, the last one
// writing dst (= base + scale * result on the final level).
template <int NF, int NT>
static void synthesis_level(fl_framelet* w, const BandPtrs& cb, const float* low, float* dst,
                            int step, const float* base, float scale, int final_, cudaStream_t s)
{
    using P = Pass<NF, NT>;
    const long long N = w->N;
    float* A = w->work;
    float* Bm = A + (long long)NF * N;
    BandPtrs ib, jb;
    for (int b = 0; b < kMaxBands; b++) ib.p[b] = jb.p[b] = nullptr;
    if (w->dim == 3) {
        P::merge(w->axes[2], pass_grid(w, NF * NF), s, cb, low, Bm, N, w->nx, w->ny, w->nz,
                 step, w->R, nullptr, 1.0f, 0);
        for (int b = 0; b < NF * NF; b++) ib.p[b] = Bm + (long long)b * N;
        P::merge(w->axes[1], pass_grid(w, NF), s, ib, nullptr, A, N, w->nx, w->ny, w->nz, step,
                 w->R, nullptr, 1.0f, 0);
        for (int b = 0; b < NF; b++) jb.p[b] = A + (long long)b * N;
        P::merge(w->axes[0], pass_grid(w, 1), s, jb, nullptr, dst, N, w->nx, w->ny, w->nz, step,
                 w->R, base, scale, final_);
    } else {
        P::merge(w->axes[1], pass_grid(w, NF), s, cb, low, A, N, w->nx, w->ny, w->nz, step,
                 w->R, nullptr, 1.0f, 0);
        for (int b = 0; b < NF; b++) jb.p[b] = A + (long long)b * N;
        P::merge(w->axes[0], pass_grid(w, 1), s, jb, nullptr, dst, N, w->nx, w->ny, w->nz, step,
                 w->R, base, scale, final_);
    }
}

// z-streaming form of a 3-D level (three-tap banks, dilation up to
// kMaxStreamStep): analysis in one kernel; synthesis as the z + x merges in
// one kernel and the y merge (with the final base + scale) streaming along y.
static bool stream_ok(const fl_framelet* w, int step)
{
    // offsets inside a plane are 32-bit byte counts
    return w->fused && w->dim == 3 && w->D.nt == 3 && step <= kMaxStreamStep &&
           (long long)w->nx * w->ny < (1LL << 30);
}

// Slices per block for `columns` blocks of one segment each, `resident` to an
// SM: the count whose whole waves read the fewest slices (two more per segment
// than it writes). 32 slices left the third wave half empty at 200 x 176 x 144
// (analysis of two levels 224 us, 204 us by this rule) and most of the chip
// idle at 77 x 61 x 45 (three levels 71 us, 32 us); at 256^3 all are alike.
static int stream_seg_len(const fl_framelet* w, int step, long long columns, int resident)
{
    const int len = class_len(w->nz, step, 0);
    const long long slots = (long long)w->sms * resident;
    int best = len;
    long long least = -1;
    for (int nseg = 1; nseg <= fl_div_up(len, 4); nseg++) {
        const int sl = fl_div_up(len, nseg);
        const long long read = (columns * nseg + slots - 1) / slots * (sl + 2);
        if (least < 0 || read < least) { least = read; best = sl; }
    }
    return best;
}

// Columns of a tile of k_syn_zx for rows longer than kRowMax: the width whose tiles
// take the least of an SM's resident threads per row (256 left 28 % of its columns
// outside rows of 600: linear bank, 600 x 40 x 300, one level 223 us, 194 with 224;
// rows of 520 82 us, 70 with 192; of 768 the same 3 x 256).
static int syn_tile(int nx, int threads)
{
    int best = 0, bp = 0, bb = 1;
    for (int t = 256; t >= 96; t -= 32) {
        const int parts = fl_div_up(nx, t), blocks = threads / (t + 32);
        if (!best || (long long)parts * bb < (long long)bp * blocks) { best = t; bp = parts; bb = blocks; }
    }
    return best;
}

template <int NF, int S>
static void ana_stream(fl_framelet* w, const float* in, const BandPtrs& cb, const BandPtrs& tb,
                       float* low_out, int last, int mode, float tau, cudaStream_t s)
{
    const unsigned gx = fl_div_up(w->nx, kSX), gy = fl_div_up(w->ny, kSY);
    // Rows that are no multiple of the 32-byte sector: neighbouring tiles share sectors
    // of every one of the 27 bands, and with three blocks an SM L2 writes them before
    // both halves are there (160 x 150 x 170: 190 us, 140 with two blocks; 180^3 219,
    // 143; 128 x 129 x 130 94, 75; 252 x 256 x 256 522, 422). Rows off 16 bytes in
    // volumes far larger than L2 do best with one (250 x 256 x 256 647, 560, 486;
    // 161 x 100 x 100 with one 64, two 60). Aligned rows want three (200^3 157, two
    // 167), as do Haar's eight bands. Unused shared memory holds the others off.
    int resident = ana_resident(NF, mode);
    size_t hold = 0;
    if (NF == 3 && mode == 0 && w->nx % 8 != 0) {
        const bool one = w->nx % 4 != 0 && w->N * 4 * w->nbands > (400LL << 20);
        hold = one ? 120000 : 76000;
        // the larger one always: the attribute is the kernel's, and another thread's
        // call between this and the launch must not lower it
        if (cudaFuncSetAttribute(k_ana_stream<NF, S, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120000) ==
            cudaSuccess)
            resident = one ? 1 : 2;
        else
            hold = 0;
    }
    const int sl = stream_seg_len(w, S, (long long)gx * gy * S, resident);
    const int nseg = fl_div_up(class_len(w->nz, S, 0), sl);
    const dim3 grid(gx, gy, (unsigned)(nseg * S));
    if (mode == 0)
        k_ana_stream<NF, S, 0><<<grid, kST, hold, s>>>(in, w->nx, w->ny, w->nz, nseg, sl, w->D, cb, tb, low_out, last, tau);
    else
        k_ana_stream<NF, S, 1><<<grid, kST, 0, s>>>(in, w->nx, w->ny, w->nz, nseg, sl, w->D, cb, tb, low_out, last, tau);
}

template <int NF, int S>
static void syn_stream(fl_framelet* w, const BandPtrs& cb, const float* low, float* dst,
                       const float* base, float scale, int final_, cudaStream_t s)
{
    const long long N = w->N;
    float* A = w->work;                                // NF arrays
    const int whole = w->nx <= kRowMax;
    const int T = whole ? 0 : syn_tile(w->nx, syn_threads(NF));
    const int W = whole ? 32 * fl_div_up(w->nx, 32) : T + 32;
    const int rows = W < 256 ? 256 / W : 1;
    const unsigned gx = whole ? 1 : fl_div_up(w->nx, T), gr = fl_div_up(w->ny, rows);
    const int sl = stream_seg_len(w, S, (long long)gx * gr * NF * S, syn_threads(NF) / (W * rows));
    const int nseg = fl_div_up(class_len(w->nz, S, 0), sl);
    k_syn_zx<NF, S><<<dim3(gx, gr, (unsigned)(nseg * NF * S)), dim3(W, rows), sizeof(float) * 2 * NF * W * rows, s>>>(
        cb, low, A, N, w->nx, w->ny, w->nz, nseg, sl, whole, w->R);
    const int nsegy = fl_div_up(class_len(w->ny, S, 0), kSegY);
    const dim3 gy(fl_div_up(w->nx, 128), w->nz, (unsigned)(nsegy * S));
    k_merge_y_stream<NF, S><<<gy, 128, 0, s>>>(A, N, dst, w->nx, w->ny, w->nz, nsegy, w->R, base,
                                               scale, final_);
}

template <int NF>
static void stream_level(fl_framelet* w, int step, bool analysis_pass, const float* in,
                         const BandPtrs& cb, const BandPtrs& tb, float* low_out, int last,
                         int mode, float tau, const float* low, float* dst, const float* base,
                         float scale, int final_, cudaStream_t s)
{
    switch (step) {
#define FL_STREAM_CASE(SS)                                                                   \
    case SS:                                                                                 \
        if (analysis_pass) ana_stream<NF, SS>(w, in, cb, tb, low_out, last, mode, tau, s);   \
        else syn_stream<NF, SS>(w, cb, low, dst, base, scale, final_, s);                    \
        break;
        FL_STREAM_CASE(1)
        FL_STREAM_CASE(2)
        FL_STREAM_CASE(4)
        FL_STREAM_CASE(8)
#undef FL_STREAM_CASE
    }
}

template <int NF, int NT>
static void run_analysis_level(fl_framelet* w, const float* in, int step, const BandPtrs& cb,
                               const BandPtrs& tb, float* low_out, int last, int mode, float tau,
                               cudaStream_t s)
{
    if constexpr (NT == 3)
        if (stream_ok(w, step)) {
            stream_level<NF>(w, step, true, in, cb, tb, low_out, last, mode, tau, nullptr,
                             nullptr, nullptr, 1.0f, 0, s);
            return;
        }
    analysis_level<NF, NT>(w, in, step, cb, tb, low_out, last, mode, tau, s);
}

template <int NF, int NT>
static void run_synthesis_level(fl_framelet* w, const BandPtrs& cb, const float* low, float* dst,
                                int step, const float* base, float scale, int final_,
                                cudaStream_t s)
{
    if constexpr (NT == 3)
        if (stream_ok(w, step)) {
            stream_level<NF>(w, step, false, nullptr, cb, cb, nullptr, 0, 0, 0.0f, low, dst,
                             base, scale, final_, s);
            return;
        }
    synthesis_level<NF, NT>(w, cb, low, dst, step, base, scale, final_, s);
}

// Analysis of all levels. mode 0: coef = W u. mode 1: Bregman update of v
// (coef argument) writing t = alpha - v_new into tcoef.
static int analysis(fl_framelet* w, const float* u, float* coef, float* tcoef, int mode,
                    float tau, cudaStream_t s)
{
    const long long N = w->N;
    float* low0 = w->work + (w->work_elems - 2 * N);
    float* low1 = low0 + N;
    const float* in = u;
    for (int l = 0; l < w->levels; l++) {
        const int step = 1 << l;
        const int last = (l == w->levels - 1) ? 1 : 0;
        float* low_out = last ? nullptr : ((l % 2 == 0) ? low0 : low1);
        BandPtrs cb = level_bands(w, coef, l), tb = level_bands(w, tcoef, l);
        if (w->kind == FL_FRAMELET_LINEAR)
            run_analysis_level<3, 3>(w, in, step, cb, tb, low_out, last, mode, tau, s);
        else if (w->kind == FL_FRAMELET_CUBIC)
            run_analysis_level<5, 5>(w, in, step, cb, tb, low_out, last, mode, tau, s);
        else
            run_analysis_level<2, 3>(w, in, step, cb, tb, low_out, last, mode, tau, s);
        int st = fl_check_launch("framelet analysis");
        if (st) return st;
        in = low_out;
    }
    return FL_OK;
}

// Synthesis: out = base + scale * W^T coef (base may be null, scale 1).
static int synthesis(fl_framelet* w, float* coef, float* out, const float* base, float scale,
                     cudaStream_t s)
{
    const long long N = w->N;
    float* low0 = w->work + (w->work_elems - 2 * N);
    float* low1 = low0 + N;
    const float* low = nullptr;
    for (int l = w->levels - 1; l >= 0; l--) {
        const int step = 1 << l;
        const int final_ = (l == 0) ? 1 : 0;
        float* dst = final_ ? out : ((l % 2 == 0) ? low0 : low1);
        BandPtrs cb = level_bands(w, coef, l);
        const float* bs = final_ ? base : nullptr;
        const float sc = final_ ? scale : 1.0f;
        if (w->kind == FL_FRAMELET_LINEAR)
            run_synthesis_level<3, 3>(w, cb, low, dst, step, bs, sc, final_, s);
        else if (w->kind == FL_FRAMELET_CUBIC)
            run_synthesis_level<5, 5>(w, cb, low, dst, step, bs, sc, final_, s);
        else
            run_synthesis_level<2, 3>(w, cb, low, dst, step, bs, sc, final_, s);
        int st = fl_check_launch("framelet synthesis");
        if (st) return st;
        low = dst;
    }
    return FL_OK;
}

extern "C" int fl_framelet_analysis(fl_framelet* w, const float* u, float* coef, void* stream)
{
    FL_RANGE("fl_framelet_analysis");
    if (!w || !u || !coef) return fl_set_error(FL_ERR_INVALID, "fl_framelet_analysis: null argument");
    int st = analysis(w, u, coef, nullptr, 0, 0.0f, (cudaStream_t)stream);
    return st ? st : fl_set_error(FL_OK, "");
}

extern "C" int fl_framelet_synthesis(fl_framelet* w, const float* coef, float* u, void* stream)
{
    FL_RANGE("fl_framelet_synthesis");
    if (!w || !u || !coef) return fl_set_error(FL_ERR_INVALID, "fl_framelet_synthesis: null argument");
    int st = synthesis(w, const_cast<float*>(coef), u, nullptr, 1.0f, (cudaStream_t)stream);
    return st ? st : fl_set_error(FL_OK, "");
}

extern "C" int fl_framelet_bregman(fl_framelet* w, const float* u, float* v, float* t,
                                   const float* Atf, float mu, float tau, float* b, void* stream)
{
    FL_RANGE("fl_framelet_bregman");
    if (!w || !u || !v || !t || !b)
        return fl_set_error(FL_ERR_INVALID, "fl_framelet_bregman: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    int st = analysis(w, u, v, t, 1, tau, s);
    if (st) return st;
    st = synthesis(w, t, b, Atf, mu, s);
    return st ? st : fl_set_error(FL_OK, "");
}

extern "C" int fl_framelet_option(fl_framelet* w, int option, int value)
{
    if (!w) return fl_set_error(FL_ERR_INVALID, "fl_framelet_option: null framelet");
    if (option != FL_FRAMELET_OPT_FUSED)
        return fl_set_error(FL_ERR_INVALID, "fl_framelet_option: unknown option %d", option);
    w->fused = value ? 1 : 0;
    return fl_set_error(FL_OK, "");
}

extern "C" int fl_framelet_shrink(fl_framelet* w, const float* coef, float* out, float tau,
                                  void* stream)
{
    if (!w || !coef || !out) return fl_set_error(FL_ERR_INVALID, "fl_framelet_shrink: null argument");
    const long long n = w->ncoef_bands * w->N;
    const long long low = w->level_base[w->levels - 1] * w->N;   // band 0 of the last level
    k_shrink<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(coef, out, n, low, low + w->N, tau);
    int st = fl_check_launch("framelet shrink");
    return st ? st : fl_set_error(FL_OK, "");
}
