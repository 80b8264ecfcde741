// Geometric Shack-Hartmann WFS on the device: gradients of the atmosphere
// seen through the DMs, upstream of the reconstruction (the geometric branch
// of cuda/wfsgrad.cu gpu_wfsgrad_iwfs with gtype_sim = 0, the reference's
// default for Shack-Hartmann WFS):
//
//   OPD(p)  = sum_atm bilinear_wrap(layer, p) - sum_dm bilinear(dm, p)
//             (cuda/accphi.cu:508 gpu_atm2loc, :556 gpu_dm2loc; the point's
//             position on a map at height h: p (1 - h/hs) + h theta - v dt isim)
//   g       = GS0 OPD                       (cuda/wfsgrad.cu:458 cuspmul)
//   g      += noise                          (cuda/wfsgrad.cu:47 add_geom_noise_do)
//
// The OPD of the WFS points is never written to memory.  A subaperture's
// average gradient is a stencil over the (nxsa+2)^2 fine-grid points around it
// (OPD points are 1/64 m, map pixels 1/5 to 1/2 m, so a window covers only a
// few pixels of each map), and the stencils have structure:
//
//   * A fully illuminated subaperture's x and y stencils are outer products of
//     two profiles (one average, one difference).  Bilinear interpolation is
//     separable too, so the gradient is a small bilinear form in the map's
//     pixels: g_x = sum_ab (A_y a)_b (D_x)_a Z_ba, where the pixel weights of
//     one axis depend only on the subaperture's column (row).  k_wfs_geom's
//     first blocks handle the subapertures of the commonest such stencil by
//     tiles of the subaperture lattice: the pixel weights of the tile's
//     columns and rows once, then a few pixels per subaperture and map.
//   * The other (partially illuminated) stencils are zero but for the window's
//     rim and the pupil edge (12% of the points): the remaining blocks keep one
//     warp per subaperture over the list of its stencil's non-zero points.
//   * A stencil with more non-zero points than a warp keeps in registers
//     (none that the reference's mkg makes) goes to k_wfs_dense, which
//     interpolates the whole window by rows.
//
// Every point of every window (the dense kernel for all) was issue-bound at
// 1,542 us for 8 instances of the 30 m system (6 WFS x 2,820 subapertures, 7
// layers + 2 DMs); by structure it takes 110 us (159 with the pixel weights
// formed pixel by pixel), and one 8 m LTAO instance 6.7 instead of 17 us.
//
// Stencils are shared by all subapertures with the same amplitude
// neighbourhood.  The noise is two standard normals per subaperture from a
// counter-based generator (Philox4x32-10, Salmon et al. 2011) keyed by the
// seed and counted by (subaperture, WFS, step, instance), so any step of any
// instance can be drawn again.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <new>
#include <utility>
#include <vector>

#include "common.cuh"

namespace mb {

constexpr int kGeomMaxWfs = 16;
constexpr int kGeomMaxScr = 16;   // atmosphere layers + DMs
constexpr int kGeomWarps = 8;     // subapertures per CTA of k_wfs_dense
constexpr int kSepTile = 8;       // subapertures across a separable tile
constexpr int kSepVec = 2 * kSepTile;  // columns, then rows, of a tile
constexpr int kSepPix = 8;        // pixels of a map a separable window spans along an axis, at most
constexpr int kSparseWarps = 4;   // subapertures per CTA of the sparse blocks
constexpr int kSepThreads = 2 * kSepTile * kSepTile;  // two threads per subaperture of a tile
constexpr int kSparsePts = 12;    // non-zero stencil points per lane
static_assert(kSepThreads == 32 * kSparseWarps, "both kinds of block share a launch");
constexpr int kGeomMaxW = 36;     // window side (nxsa + 2)
constexpr int kGeomRows = 17;    // window rows per band (OPD in registers)
constexpr int kGeomTail = (kGeomRows * (kGeomMaxW - 32) + 31) / 32;  // points of columns >= 32 per lane
constexpr int kGeomBlk = 16;     // layer pixels a window spans across, at most
constexpr int kGeomBlkStride = kGeomBlk + 1;
constexpr int kGeomHStride = kGeomMaxW;
constexpr double kGeomMaxStep = (kGeomBlk - 3.0) / (kGeomMaxW - 1.0);  // layer pixels per fine-grid step
// shared-memory bounds the kernel relies on: a band's pixel block is at most
// kGeomBlk x kGeomBlk, its interpolated rows fit the kGeomBlk x kGeomHStride
// table, and a tail point's band row fits the 8 bits it is packed in
static_assert(kGeomMaxStep * (kGeomMaxW - 1) + 3 <= kGeomBlk, "window wider than the pixel block");
static_assert(kGeomRows <= kGeomMaxW && kGeomRows < 256, "band rows");

struct GeomScr {
    const float *p;    // [ny][nx], x fastest
    long inst_stride;  // floats between instances (0: shared)
    int nx, ny;
    float alpha;
    int wrap;
};
struct GeomWfsT {
    int nsa, nxsa, sa_off;
    long g_off;
    // subapertures of the separable stencil: tiles of the lattice of their
    // columns and rows (offsets into GeomLists)
    int ntile, tile_off, ncol, nrow, col_off, row_off, grid_off, prof_off;
    float cx, cy;                 // the separable stencils' response to a constant OPD
    int nsparse, sparse_off;      // subapertures of the sparse list
    int ndense, dense_off;        // and of the dense one
};
// Index lists of every WFS, concatenated (device).
struct GeomLists {
    const int *tile;     // x tile | y tile << 16
    const int *col, *row;  // fine-grid index of each lattice column's, row's first point
    const int *grid;     // [nrow][ncol] subaperture at a lattice place, -1: none
    const float *prof;   // per WFS [4][nxsa + 2]: x stencil along y, along x, y stencil along x, along y
    const int2 *sa;      // subapertures of the sparse and the dense lists, and their stencils' point lists
    const int *pt_off;   // start of each point list (one past the last: the end)
    const int *pt;       // non-zero points: window row << 8 | column
    const float2 *ptw;   // and x, y weights
};
struct GeomCoef {  // screen index = fine-grid index * s + b (before the wind shift)
    double sx, bx, sy, by;
};
struct GeomTab {
    int nwfs, nscr, natm;
    GeomWfsT w[kGeomMaxWfs];
    GeomScr s[kGeomMaxScr];
    GeomCoef c[kGeomMaxWfs][kGeomMaxScr];
};

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const unsigned lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const unsigned lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

// A map's position of a window's first point along one axis: the integer part
// (wrapped for the atmosphere) and the fraction.
__device__ __forceinline__ void geom_base(const GeomScr &S, int g0, double s, double b, double shift, int n, int &i0,
                                          float &f0) {
    const double u = fma((double)g0, s, b) - shift;
    const double fu = floor(u);
    long long iu = (long long)fmin(fmax(fu, -1e9), 1e9);
    if (S.wrap) {
        iu %= n;
        if (iu < 0) iu += n;
    }
    i0 = (int)iu;
    f0 = (float)(u - fu);
}

// The two gradients of one subaperture, with their noise when seed is not 0.
__device__ __forceinline__ void geom_store(const GeomWfsT &W, int isa, int iw, int inst, float gx, float gy,
                                           const float *__restrict__ nea, float *__restrict__ grad, long grad_stride,
                                           long isim, unsigned long long seed) {
    if (seed) {
        const uint4 o = philox4x32_10(make_uint4((unsigned)isa, (unsigned)iw, (unsigned)isim, (unsigned)inst),
                                      make_uint2((unsigned)seed, (unsigned)(seed >> 32)));
        const double u1 = ((double)o.x + 1.0) * 0x1p-32, u2 = (double)o.y * 0x1p-32;
        const double rr = sqrt(-2.0 * log(u1));
        double sn, cs;
        sincospi(2.0 * u2, &sn, &cs);
        const float n1 = (float)(rr * cs), n2 = (float)(rr * sn);
        const float *ne = nea + 3L * W.sa_off;
        gx = fmaf(n1, ne[isa], gx);
        gy = fmaf(n2, ne[W.nsa + isa], fmaf(n1, ne[2 * W.nsa + isa], gy));
    }
    float *g = grad + (long)inst * grad_stride + W.g_off;
    g[isa] = gx;
    g[W.nsa + isa] = gy;
}

struct SepShared {
    int i0[kGeomMaxScr][kSepVec];
    float f0[kGeomMaxScr][kSepVec];
    float2 w[kGeomMaxScr][kSepVec][kSepPix + 1];  // (average, difference) pixel weights; odd stride: no conflicts
    float prof[4][kGeomMaxW];
};
struct SparseShared {
    int4 base[kSparseWarps][kGeomMaxScr];
    float blk[kSparseWarps][kGeomBlk * kGeomBlkStride];
};

// One tile of the separable subapertures (kSepThreads threads).  The pixel
// weights of an axis are sums of the profile over the window's points, by a
// thread per (map, column or row); a subaperture then needs nbu x nbv pixels of each map, split
// over two threads by rows.  The block's first pixel is subtracted from the
// others (its share is the stencil's response to a constant, 0 for a gradient)
// so that the differences, not the OPD itself, meet FP32 rounding.
__device__ __forceinline__ void sep_tile(const GeomTab &t, const GeomLists &L, SepShared &sh, int tile, int iw,
                                         int inst, const float *__restrict__ nea,
                                         const double2 *__restrict__ wind_px, float *__restrict__ grad,
                                         long grad_stride, long isim, unsigned long long seed) {
    const GeomWfsT &W = t.w[iw];
    const int wn = W.nxsa + 2;
    const int tt = L.tile[W.tile_off + tile];
    const int c0 = (tt & 0xffff) * kSepTile, r0 = (tt >> 16) * kSepTile;
    for (int e = threadIdx.x; e < 4 * wn; e += kSepThreads) sh.prof[e / wn][e % wn] = L.prof[W.prof_off + e];
    __syncthreads();
    for (int e = threadIdx.x; e < t.nscr * kSepVec; e += kSepThreads) {
        const int s = e / kSepVec, v = e - s * kSepVec;
        const bool isx = v < kSepTile;
        const int q = isx ? min(c0 + v, W.ncol - 1) : min(r0 + v - kSepTile, W.nrow - 1);
        const int g0 = (isx ? L.col[W.col_off + q] : L.row[W.row_off + q]) - 1;
        const GeomCoef c = t.c[iw][s];
        double shift = 0;
        if (s < t.natm) {  // frozen flow: the layer moves by v dt per step
            const double2 w = wind_px[(long)inst * t.natm + s];
            shift = (isx ? w.x : w.y) * (double)isim;
        }
        const int n = isx ? t.s[s].nx : t.s[s].ny;
        int i0;
        float f0;
        geom_base(t.s[s], g0, isx ? c.sx : c.sy, isx ? c.bx : c.by, shift, n, i0, f0);
        sh.i0[s][v] = i0;
        sh.f0[s][v] = f0;
        // walk the window's points: each counts for the pixel before it and the
        // next (points move less than a pixel), complete once the walk passes it
        const float step = (float)(isx ? c.sx : c.sy);
        const float *pa = sh.prof[isx ? 2 : 0], *pd = sh.prof[isx ? 1 : 3];
        float2 *w = sh.w[s][v];
        float2 w0 = make_float2(0.f, 0.f), w1 = w0;
        int k = 0;
        for (int p = 0; p < wn; p++) {
            const float u = fmaf((float)p, step, f0), fl = floorf(u);
            if ((int)fl > k) {
                w[k++] = w0;
                w0 = w1;
                w1 = make_float2(0.f, 0.f);
            }
            if (t.s[s].wrap || (i0 + k >= 0 && i0 + k < n)) {  // off the map: no contribution
                const float a1 = u - fl, a0 = 1.f - a1;
                w0.x = fmaf(pa[p], a0, w0.x);
                w0.y = fmaf(pd[p], a0, w0.y);
                w1.x = fmaf(pa[p], a1, w1.x);
                w1.y = fmaf(pd[p], a1, w1.y);
            }
        }
        w[k] = w0;
        w[k + 1] = w1;
        for (int q = k + 2; q < kSepPix; q++) w[q] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int h = threadIdx.x & 1, sub = threadIdx.x >> 1;
    const int i = sub % kSepTile, j = sub / kSepTile;
    const bool in = c0 + i < W.ncol && r0 + j < W.nrow;
    const int isa = in ? L.grid[W.grid_off + (r0 + j) * W.ncol + c0 + i] : -1;
    float gx = 0.f, gy = 0.f;
    if (isa >= 0) {
        for (int s = 0; s < t.nscr; s++) {
            const GeomScr S = t.s[s];
            const float *__restrict__ P = S.p + (long)inst * S.inst_stride;
            const int iu = sh.i0[s][i], iv = sh.i0[s][kSepTile + j];
            const float2 *wu = sh.w[s][i], *wv = sh.w[s][kSepTile + j];
            const int nbu = (int)fmaf((float)(wn - 1), (float)t.c[iw][s].sx, sh.f0[s][i]) + 2;
            const int nbv = (int)fmaf((float)(wn - 1), (float)t.c[iw][s].sy, sh.f0[s][kSepTile + j]) + 2;
            // the whole block on the map (always, for a wrapped one)
            const bool inside = S.wrap || (iu >= 0 && iu + nbu <= S.nx && iv >= 0 && iv + nbv <= S.ny);
            const float z0 = inside ? __ldg(P + (long)iv * S.nx + iu) : 0.f;
            float mx = 0.f, my = 0.f;
            for (int bv = h; bv < nbv; bv += 2) {
                int r = iv + bv;
                r -= (S.wrap ? r >= S.ny : r == S.ny) ? S.ny : 0;  // the +1 neighbour of the last row is row 0
                const bool rok = S.wrap || (r >= 0 && r < S.ny);
                float ta = 0.f, td = 0.f;
                for (int b0 = 0; b0 < nbu; b0 += 4) {
                    float z[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        int c = iu + b0 + q;
                        c -= (S.wrap ? c >= S.nx : c == S.nx) ? S.nx : 0;
                        z[q] = b0 + q < nbu && rok && c >= 0 && c < S.nx ? __ldg(P + (long)r * S.nx + c) - z0 : 0.f;
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float2 w = wu[min(b0 + q, kSepPix - 1)];
                        ta = fmaf(w.x, z[q], ta);
                        td = fmaf(w.y, z[q], td);
                    }
                }
                mx = fmaf(wv[bv].x, td, mx);
                my = fmaf(wv[bv].y, ta, my);
            }
            if (h == 0) {
                mx = fmaf(W.cx, z0, mx);
                my = fmaf(W.cy, z0, my);
            }
            gx = fmaf(S.alpha, mx, gx);
            gy = fmaf(S.alpha, my, gy);
        }
    }
    gx += __shfl_xor_sync(0xffffffffu, gx, 1);
    gy += __shfl_xor_sync(0xffffffffu, gy, 1);
    if (isa >= 0 && h == 0) geom_store(W, isa, iw, inst, gx, gy, nea, grad, grad_stride, isim, seed);
}

// One warp per subaperture over the non-zero points of its stencil: each map's
// pixel block staged in shared memory, the OPD of kSparsePts points per lane
// in registers.
__device__ __forceinline__ void sparse_sa(const GeomTab &t, const GeomLists &L, SparseShared &sh, int k, int iw,
                                          int inst, const int *__restrict__ sa_ix, const int *__restrict__ sa_iy,
                                          const float *__restrict__ nea, const double2 *__restrict__ wind_px,
                                          float *__restrict__ grad, long grad_stride, long isim,
                                          unsigned long long seed) {
    const GeomWfsT &W = t.w[iw];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= W.nsparse) return;  // the whole warp: no block-wide barrier here
    const int2 ent = L.sa[W.sparse_off + k];
    const int isa = ent.x, gi = W.sa_off + isa;
    const int wn = W.nxsa + 2;
    if (lane < t.nscr) {
        const GeomCoef c = t.c[iw][lane];
        double2 w = make_double2(0, 0);
        if (lane < t.natm) w = wind_px[(long)inst * t.natm + lane];
        int4 b;
        float fu, fv;
        geom_base(t.s[lane], sa_ix[gi] - 1, c.sx, c.bx, w.x * (double)isim, t.s[lane].nx, b.x, fu);
        geom_base(t.s[lane], sa_iy[gi] - 1, c.sy, c.by, w.y * (double)isim, t.s[lane].ny, b.y, fv);
        b.z = __float_as_int(fu);
        b.w = __float_as_int(fv);
        sh.base[wid][lane] = b;
    }
    __syncwarp();
    float *blk = sh.blk[wid];
    const int p0 = L.pt_off[ent.y], npt = L.pt_off[ent.y + 1] - p0;
    float opd[kSparsePts], pc[kSparsePts], pr[kSparsePts];
#pragma unroll
    for (int q = 0; q < kSparsePts; q++) {
        const int e = lane + 32 * q;
        const int rc = e < npt ? L.pt[p0 + e] : 0;
        pc[q] = (float)(rc & 255);
        pr[q] = (float)(rc >> 8);
        opd[q] = 0.f;
    }
    for (int s = 0; s < t.nscr; s++) {
        const GeomScr S = t.s[s];
        const int4 b = sh.base[wid][s];
        const float sxf = (float)t.c[iw][s].sx, syf = (float)t.c[iw][s].sy;
        const float fu0 = __int_as_float(b.z), fv0 = __int_as_float(b.w);
        const float *__restrict__ P = S.p + (long)inst * S.inst_stride;
        const int nbu = min((int)fmaf((float)(wn - 1), sxf, fu0) + 2, kGeomBlk);
        const int nbv = min((int)fmaf((float)(wn - 1), syf, fv0) + 2, kGeomBlk);
        const float inv_nbu = __frcp_rn((float)nbu);
        __syncwarp();  // the previous map's block is no longer read
        for (int e = lane; e < nbu * nbv; e += 32) {
            const int bv = (int)(((float)e + 0.5f) * inv_nbu), bu = e - bv * nbu;
            int c = b.x + bu, r = b.y + bv;
            c -= (S.wrap ? c >= S.nx : c == S.nx) ? S.nx : 0;  // the +1 neighbour of the last column is column 0
            r -= (S.wrap ? r >= S.ny : r == S.ny) ? S.ny : 0;
            blk[bv * kGeomBlkStride + bu] =
                c >= 0 && c < S.nx && r >= 0 && r < S.ny ? __ldg(P + (long)r * S.nx + c) : 0.f;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kSparsePts; q++) {
            if (32 * q >= npt) break;  // lanes past the end repeat point 0 and have no weight
            const float u = fmaf(pc[q], sxf, fu0), v = fmaf(pr[q], syf, fv0);
            const float fu = floorf(u), fv = floorf(v), ax = u - fu, ay = v - fv;
            const int lu = (int)fu, lv = (int)fv;
            const float *m = blk + lv * kGeomBlkStride + lu;
            const float h0 = fmaf(m[1] - m[0], ax, m[0]);
            const float h1 = fmaf(m[kGeomBlkStride + 1] - m[kGeomBlkStride], ax, m[kGeomBlkStride]);
            const float val = fmaf(h1 - h0, ay, h0);
            const bool ok = S.wrap || (b.x + lu >= 0 && b.x + lu < S.nx && b.y + lv >= 0 && b.y + lv < S.ny);
            if (ok) opd[q] = fmaf(S.alpha, val, opd[q]);  // off the map: no contribution
        }
    }
    float gx = 0.f, gy = 0.f;
#pragma unroll
    for (int q = 0; q < kSparsePts; q++) {
        const int e = lane + 32 * q;
        if (e < npt) {
            const float2 w = L.ptw[p0 + e];
            gx = fmaf(w.x, opd[q], gx);
            gy = fmaf(w.y, opd[q], gy);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gx += __shfl_xor_sync(0xffffffffu, gx, o);
        gy += __shfl_xor_sync(0xffffffffu, gy, o);
    }
    if (lane == 0) geom_store(W, isa, iw, inst, gx, gy, nea, grad, grad_stride, isim, seed);
}

// grid: (max over WFS of tiles + ceil(sparse / kSparseWarps), nwfs, nbatch); block: kSepThreads.
// sa_ix/sa_iy: fine-grid index of each subaperture's first point; nea per WFS
// [3][nsa] (sqrt-NEA xx, yy, xy) at 3*sa_off; wind_px: per instance and
// atmosphere layer, the shift in layer pixels per step (v dt / dx).
__global__ void __launch_bounds__(kSepThreads)
k_wfs_geom(const __grid_constant__ GeomTab t, const __grid_constant__ GeomLists L, const int *__restrict__ sa_ix,
           const int *__restrict__ sa_iy, const float *__restrict__ nea, const double2 *__restrict__ wind_px,
           float *__restrict__ grad, long grad_stride, long isim, unsigned long long seed) {
    __shared__ union {
        SepShared sep;
        SparseShared sparse;
    } sh;
    const int iw = blockIdx.y, inst = blockIdx.z, nt = t.w[iw].ntile;
    if ((int)blockIdx.x < nt)
        sep_tile(t, L, sh.sep, blockIdx.x, iw, inst, nea, wind_px, grad, grad_stride, isim, seed);
    else
        sparse_sa(t, L, sh.sparse, (blockIdx.x - nt) * kSparseWarps + (threadIdx.x >> 5), iw, inst, sa_ix, sa_iy, nea,
                  wind_px, grad, grad_stride, isim, seed);
}

// The window of every point (dense stencils), one warp per subaperture of the
// dense list.  grid: (ceil(max dense / kGeomWarps), nwfs, nbatch); block:
// kGeomWarps warps.  sa_st: each subaperture's stencil; st_off: the offset of
// each stencil ([2][W*W] floats) in st.
__global__ void __launch_bounds__(kGeomWarps * 32, 4)
k_wfs_dense(const __grid_constant__ GeomTab t, const __grid_constant__ GeomLists L, const int *__restrict__ sa_ix,
            const int *__restrict__ sa_iy, const int *__restrict__ sa_st, const float *__restrict__ st,
            const long *__restrict__ st_off, const float *__restrict__ nea, const double2 *__restrict__ wind_px,
            float *__restrict__ grad, long grad_stride, long isim, unsigned long long seed) {
    __shared__ int4 sbase[kGeomWarps][kGeomMaxScr];
    __shared__ float sblk[kGeomWarps][kGeomBlk * kGeomBlkStride];
    __shared__ float shx[kGeomWarps][kGeomBlk * kGeomHStride];
    __shared__ float2 srow[kGeomWarps][kGeomRows];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int iw = blockIdx.y, inst = blockIdx.z;
    const GeomWfsT &W = t.w[iw];
    const int k = blockIdx.x * kGeomWarps + wid;
    if (k >= W.ndense) return;  // the whole warp: no block-wide barrier below
    const int isa = L.sa[W.dense_off + k].x, gi = W.sa_off + isa;
    const int wn = W.nxsa + 2, npts = wn * wn;
    const int gx0 = sa_ix[gi] - 1, gy0 = sa_iy[gi] - 1;
    // each map's position of the window's first point: integer part (wrapped
    // for the atmosphere) and fraction
    if (lane < t.nscr) {
        const GeomCoef c = t.c[iw][lane];
        double2 w = make_double2(0, 0);
        if (lane < t.natm) w = wind_px[(long)inst * t.natm + lane];  // frozen flow: the layer moves by v dt per step
        int4 b;
        float fu, fv;
        geom_base(t.s[lane], gx0, c.sx, c.bx, w.x * (double)isim, t.s[lane].nx, b.x, fu);
        geom_base(t.s[lane], gy0, c.sy, c.by, w.y * (double)isim, t.s[lane].ny, b.y, fv);
        b.z = __float_as_int(fu);
        b.w = __float_as_int(fv);
        sbase[wid][lane] = b;
    }
    __syncwarp();
    const float *__restrict__ w = st + st_off[sa_st[gi]];
    float *blk = sblk[wid], *hx = shx[wid];
    float gx = 0.f, gy = 0.f;
    // Lane c owns window column c (< 32) of a band of kGeomRows rows; the
    // points of the columns from 32 on (wn > 32: at most 4 columns) are dealt
    // out over the lanes, kGeomTail at most each.  OPD of the band stays in
    // registers.
    const int ntail = wn > 32 ? wn - 32 : 0;
    const bool main_ok = lane < wn;
    for (int r0 = 0; r0 < wn; r0 += kGeomRows) {
        const int nr = min(kGeomRows, wn - r0);
        float opd[kGeomRows];
#pragma unroll
        for (int j = 0; j < kGeomRows; j++) opd[j] = 0.f;
        float opdt[kGeomTail];
        int tpk[kGeomTail];  // band row << 8 | column of each tail point, -1: none
#pragma unroll
        for (int q = 0; q < kGeomTail; q++) {
            const int tp = lane + 32 * q;
            opdt[q] = 0.f;
            tpk[q] = tp < nr * ntail ? (tp / ntail) << 8 | (32 + tp % ntail) : -1;
        }
        for (int s = 0; s < t.nscr; s++) {
            const GeomScr S = t.s[s];
            const int4 b = sbase[wid][s];
            const float sxf = (float)t.c[iw][s].sx, syf = (float)t.c[iw][s].sy;
            const float fu0 = __int_as_float(b.z), fv0 = __int_as_float(b.w);
            const float *__restrict__ P = S.p + (long)inst * S.inst_stride;
            // the layer pixels this band touches: columns 0..nbu-1 and rows
            // v0..v0+nbv-1 from the window origin's pixel (the +1 neighbours included)
            const int v0 = (int)floorf(fmaf((float)r0, syf, fv0));
            const int nbv = min((int)floorf(fmaf((float)(r0 + nr - 1), syf, fv0)) + 2 - v0, kGeomBlk);
            const int nbu = min((int)floorf(fmaf((float)(wn - 1), sxf, fu0)) + 2, kGeomBlk);
            const float inv_nbu = __frcp_rn((float)nbu);
            __syncwarp();  // the previous map's tables are no longer read
            for (int e = lane; e < nbu * nbv; e += 32) {
                const int bv = (int)(((float)e + 0.5f) * inv_nbu), bu = e - bv * nbu;
                int c = b.x + bu, r = b.y + v0 + bv;
                float val = 0.f;
                if (S.wrap) {
                    c -= c >= S.nx ? S.nx : 0;
                    r -= r >= S.ny ? S.ny : 0;
                    val = __ldg(P + (long)r * S.nx + c);
                } else {
                    c = c == S.nx ? 0 : c;  // the +1 neighbour of the last column is column 0
                    r = r == S.ny ? 0 : r;
                    if (c >= 0 && c < S.nx && r >= 0 && r < S.ny) val = __ldg(P + (long)r * S.nx + c);
                }
                blk[bv * kGeomBlkStride + bu] = val;
            }
            __syncwarp();
            // each block row interpolated along x at every window column
            for (int cc = lane; cc < wn; cc += 32) {
                const float uf = fmaf((float)cc, sxf, fu0), fl = floorf(uf), ax = uf - fl;
                const int lu = (int)fl;
                const bool ok = S.wrap || (b.x + lu >= 0 && b.x + lu < S.nx);  // off the map: no contribution
                for (int bv = 0; bv < nbv; bv++) {
                    const float m0 = blk[bv * kGeomBlkStride + lu], m1 = blk[bv * kGeomBlkStride + lu + 1];
                    hx[bv * kGeomHStride + cc] = ok ? fmaf(m1 - m0, ax, m0) : 0.f;
                }
            }
            // each band row's pair of interpolated rows (offset in hx, -1 when
            // the row is off the map) and its fraction along y
            for (int rr = lane; rr < nr; rr += 32) {  // every band row, whatever kGeomRows is
                const float vf = fmaf((float)(r0 + rr), syf, fv0), flv = floorf(vf);
                const int lv = (int)flv - v0;
                const bool rok = S.wrap || (b.y + (int)flv >= 0 && b.y + (int)flv < S.ny);
                srow[wid][rr] = make_float2(__int_as_float(rok && lv >= 0 && lv + 1 < nbv ? lv * kGeomHStride : -1),
                                            vf - flv);
            }
            __syncwarp();
            // every point of the band: along y between two of those rows
#pragma unroll
            for (int j = 0; j < kGeomRows; j++) {
                if (j < nr && main_ok) {
                    const float2 q = srow[wid][j];
                    const int off = __float_as_int(q.x);
                    if (off >= 0) {
                        const float h0 = hx[off + lane], h1 = hx[off + kGeomHStride + lane];
                        opd[j] = fmaf(S.alpha, fmaf(h1 - h0, q.y, h0), opd[j]);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < kGeomTail; q++) {
                if (tpk[q] >= 0) {
                    const int tc = tpk[q] & 255;
                    const float2 rq = srow[wid][tpk[q] >> 8];
                    const int off = __float_as_int(rq.x);
                    if (off >= 0) {
                        const float h0 = hx[off + tc], h1 = hx[off + kGeomHStride + tc];
                        opdt[q] = fmaf(S.alpha, fmaf(h1 - h0, rq.y, h0), opdt[q]);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kGeomRows; j++) {
            if (j < nr && main_ok) {
                const int k = (r0 + j) * wn + lane;
                gx = fmaf(__ldg(w + k), opd[j], gx);
                gy = fmaf(__ldg(w + npts + k), opd[j], gy);
            }
        }
#pragma unroll
        for (int q = 0; q < kGeomTail; q++) {
            if (tpk[q] >= 0) {
                const int k = (r0 + (tpk[q] >> 8)) * wn + (tpk[q] & 255);
                gx = fmaf(__ldg(w + k), opdt[q], gx);
                gy = fmaf(__ldg(w + npts + k), opdt[q], gy);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gx += __shfl_xor_sync(0xffffffffu, gx, o);
        gy += __shfl_xor_sync(0xffffffffu, gy, o);
    }
    if (lane == 0) geom_store(W, isa, iw, inst, gx, gy, nea, grad, grad_stride, isim, seed);
}

struct GeomWfsHost {
    int nwfs = 0, natm = 0, ndm = 0, nbatch = 1;
    long ngrad = 0, nact = 0, atm_stride = 0;
    double dt = 0;
    std::vector<int> nsa, nxsa;
    std::vector<double> dx, gox, goy, thetax, thetay, hs;
    std::vector<int> anx, any;
    std::vector<double> adx, aox, aoy, aht;
    std::vector<double> wind;  // [nbatch][natm][2] m/s
    std::vector<long> aoff;  // layer offsets within one instance
    std::vector<int> dnx, dny;
    std::vector<double> ddx, dox, doy, dht;
    std::vector<long> doff;  // DM offsets within one instance's commands
    DevBuf<int> sa_ix, sa_iy, sa_st;
    DevBuf<float> st, nea, atm;
    DevBuf<double2> wind_px;
    void upload_wind() {
        std::vector<double2> w((size_t)nbatch * natm);
        for (int i = 0; i < nbatch; i++)
            for (int l = 0; l < natm; l++) {
                const size_t k = (size_t)i * natm + l;
                w[k] = make_double2(wind[2 * k] * dt / adx[l], wind[2 * k + 1] * dt / adx[l]);
            }
        wind_px.upload(w);
    }
    DevBuf<long> st_off;
    bool have_nea = false;
    // the subapertures by kind of stencil (GeomLists), and each WFS's part of them
    std::vector<GeomWfsT> parts;
    DevBuf<int> l_tile, l_col, l_row, l_grid, l_ptoff, l_pt;
    DevBuf<int2> l_sa;
    DevBuf<float> l_prof;
    DevBuf<float2> l_ptw;
    int max_blocks = 0, max_dense = 0;
    GeomLists lists() const {
        return GeomLists{l_tile.p, l_col.p, l_row.p, l_grid.p, l_prof.p, l_sa.p, l_ptoff.p, l_pt.p, l_ptw.p};
    }
    void build_lists(const std::vector<int> &ix, const std::vector<int> &iy, const std::vector<int> &sid,
                     const std::vector<long> &soff, const double *st);
};

// Whether the n x n array w is a[row] * b[col] to well below FP32 rounding of
// its largest entry, and the profiles.
static bool outer_product(const double *w, int n, std::vector<double> &a, std::vector<double> &b) {
    int best = 0;
    for (int k = 0; k < n * n; k++)
        if (std::fabs(w[k]) > std::fabs(w[best])) best = k;
    const int r0 = best / n, c0 = best % n;
    const double big = w[best];
    if (!(std::fabs(big) > 0) || !std::isfinite(big)) return false;
    a.resize(n);
    b.resize(n);
    for (int k = 0; k < n; k++) {
        a[k] = w[k * n + c0] / big;
        b[k] = w[r0 * n + k];
    }
    for (int r = 0; r < n; r++)
        for (int c = 0; c < n; c++)
            if (!(std::fabs(w[r * n + c] - a[r] * b[c]) <= 1e-10 * std::fabs(big))) return false;
    return true;
}

// Sort every WFS's subapertures by how their gradients are computed: the
// commonest separable stencil by tiles of the lattice its subapertures form,
// the others by their stencil's non-zero points, and stencils with more points
// than a warp holds by whole windows.  The separable form needs every map's
// window within kSepPix pixels, and a lattice that the subapertures fill to a
// quarter at least (a tile's weights pay when most of its places are taken).
void GeomWfsHost::build_lists(const std::vector<int> &ix, const std::vector<int> &iy, const std::vector<int> &sid,
                              const std::vector<long> &soff, const double *stv) {
    std::vector<int> tile, col, row, grid, ptoff{0}, pt;
    std::vector<int2> sa;
    std::vector<float> prof;
    std::vector<float2> ptw;
    std::map<std::pair<int, int>, int> point_list;  // of a stencil at a window size
    auto points = [&](int k, int wn) {
        const auto f = point_list.emplace(std::make_pair(k, wn), (int)ptoff.size() - 1);
        if (f.second) {
            const double *w = stv + soff[k];
            for (int e = 0; e < wn * wn; e++)
                if (w[e] != 0 || w[wn * wn + e] != 0) {
                    pt.push_back((e / wn) << 8 | (e % wn));
                    ptw.push_back(make_float2((float)w[e], (float)w[wn * wn + e]));
                }
            ptoff.push_back((int)pt.size());
        }
        return f.first->second;
    };
    std::vector<int2> dense_sa;
    parts.assign(nwfs, GeomWfsT{});
    int base = 0;
    long goff = 0;
    for (int i = 0; i < nwfs; base += nsa[i], goff += 2L * nsa[i], i++) {
        GeomWfsT &P = parts[i];
        const int wn = nxsa[i] + 2;
        P.nsa = nsa[i];
        P.nxsa = nxsa[i];
        P.sa_off = base;
        P.g_off = goff;
        bool narrow = true;
        for (int s = 0; s < natm + ndm; s++) {
            const double ht = s < natm ? aht[s] : dht[s - natm], sdx = s < natm ? adx[s] : ddx[s - natm];
            const double sc = std::isfinite(hs[i]) ? 1.0 - ht / hs[i] : 1.0;
            if (std::floor(1.001 + (wn - 1) * dx[i] * sc / sdx) + 2 > kSepPix) narrow = false;
        }
        std::map<int, int> use;
        for (int j = 0; j < nsa[i]; j++) use[sid[base + j]]++;
        int sep = -1;
        std::vector<double> xa, xb, ya, yb, ta, tb, ua, ub;
        for (const auto &u : use)
            if (narrow && (sep < 0 || u.second > use[sep]) && outer_product(stv + soff[u.first], wn, ta, tb) &&
                outer_product(stv + soff[u.first] + wn * wn, wn, ua, ub)) {
                sep = u.first;
                xa = ta, xb = tb, ya = ua, yb = ub;
            }
        std::vector<int> cols, rows, take(nsa[i], 0);
        if (sep >= 0) {
            for (int j = 0; j < nsa[i]; j++)
                if (sid[base + j] == sep) {
                    cols.push_back(ix[base + j]);
                    rows.push_back(iy[base + j]);
                }
            for (auto *v : {&cols, &rows}) {
                std::sort(v->begin(), v->end());
                v->erase(std::unique(v->begin(), v->end()), v->end());
            }
        }
        const long places = (long)cols.size() * (long)rows.size();
        if (sep >= 0 && places <= 4L * use[sep] && cols.size() < 65536 && rows.size() < 65536) {
            P.ncol = (int)cols.size();
            P.nrow = (int)rows.size();
            P.col_off = (int)col.size();
            P.row_off = (int)row.size();
            P.grid_off = (int)grid.size();
            P.prof_off = (int)prof.size();
            P.tile_off = (int)tile.size();
            std::vector<int> g((size_t)places, -1);
            for (int j = 0; j < nsa[i]; j++) {
                if (sid[base + j] != sep) continue;
                const int c = (int)(std::lower_bound(cols.begin(), cols.end(), ix[base + j]) - cols.begin());
                const int r = (int)(std::lower_bound(rows.begin(), rows.end(), iy[base + j]) - rows.begin());
                int &at = g[(size_t)r * P.ncol + c];
                if (at >= 0) continue;  // a second subaperture at one place: by its points
                at = j;
                take[j] = 1;
            }
            for (int r = 0; r < P.nrow; r += kSepTile)
                for (int c = 0; c < P.ncol; c += kSepTile) {
                    bool any = false;
                    for (int y = r; y < std::min(P.nrow, r + kSepTile); y++)
                        for (int x = c; x < std::min(P.ncol, c + kSepTile); x++)
                            any = any || g[(size_t)y * P.ncol + x] >= 0;
                    if (any) tile.push_back(c / kSepTile | (r / kSepTile) << 16);
                }
            P.ntile = (int)tile.size() - P.tile_off;
            col.insert(col.end(), cols.begin(), cols.end());
            row.insert(row.end(), rows.begin(), rows.end());
            grid.insert(grid.end(), g.begin(), g.end());
            double sum[4] = {0, 0, 0, 0};
            int q = 0;
            for (const auto *v : {&xa, &xb, &yb, &ya}) {
                for (double e : *v) {
                    prof.push_back((float)e);
                    sum[q] += e;
                }
                q++;
            }
            P.cx = (float)(sum[0] * sum[1]);
            P.cy = (float)(sum[2] * sum[3]);
        }
        P.sparse_off = (int)sa.size();
        dense_sa.clear();
        for (int j = 0; j < nsa[i]; j++) {
            if (take[j]) continue;
            const int k = points(sid[base + j], wn);
            (ptoff[k + 1] - ptoff[k] <= 32 * kSparsePts ? sa : dense_sa).push_back(make_int2(j, k));
        }
        P.nsparse = (int)sa.size() - P.sparse_off;
        P.dense_off = (int)sa.size();
        P.ndense = (int)dense_sa.size();
        sa.insert(sa.end(), dense_sa.begin(), dense_sa.end());
        max_blocks = std::max(max_blocks, P.ntile + (P.nsparse + kSparseWarps - 1) / kSparseWarps);
        max_dense = std::max(max_dense, P.ndense);
    }
    l_tile.upload(tile);
    l_col.upload(col);
    l_row.upload(row);
    l_grid.upload(grid);
    l_prof.upload(prof);
    l_sa.upload(sa);
    l_ptoff.upload(ptoff);
    l_pt.upload(pt);
    l_ptw.upload(ptw);
}

}  // namespace mb

struct mb_geom_wfs {
    mb::GeomWfsHost H;
};

extern "C" {

int mb_geom_wfs_create(const mb_geom_wfs_desc *d, mb_geom_wfs **out) {
    using namespace mb;
    if (!out || !d || d->nwfs < 1 || d->nwfs > kGeomMaxWfs || d->natm < 0 || d->ndm < 0 ||
        d->natm + d->ndm > kGeomMaxScr || d->nbatch < 1 || !d->nsa || !d->nxsa || !d->dx || !d->gox || !d->goy ||
        !d->thetax || !d->thetay || !d->hs || !d->sa_ix || !d->sa_iy || !d->sa_stencil || d->nstencil < 1 ||
        !d->stencil_off || !d->stencils || d->stencil_len < 1 ||
        (d->natm && (!d->atm_nx || !d->atm_ny || !d->atm_dx || !d->atm_ox || !d->atm_oy || !d->atm_ht ||
                     !d->atm_vx || !d->atm_vy)) ||
        (d->ndm && (!d->dm_nx || !d->dm_ny || !d->dm_dx || !d->dm_ox || !d->dm_oy || !d->dm_ht))) {
        set_error("mb_geom_wfs_create: invalid descriptor");
        return MB_EINVAL;
    }
    *out = nullptr;
    mb_geom_wfs *h = new (std::nothrow) mb_geom_wfs();
    if (!h) return MB_ENOMEM;
    try {
        GeomWfsHost &H = h->H;
        H.nwfs = d->nwfs;
        H.natm = d->natm;
        H.ndm = d->ndm;
        H.nbatch = d->nbatch;
        H.dt = d->dt;
        long nsa_tot = 0;
        for (int i = 0; i < d->nwfs; i++) {
            if (d->nsa[i] < 1 || d->nxsa[i] < 1 || d->nxsa[i] + 2 > kGeomMaxW || !(d->dx[i] > 0)) {
                set_error("mb_geom_wfs_create: WFS %d: nsa %d, nxsa %d (window at most %d points across)", i,
                          d->nsa[i], d->nxsa[i], kGeomMaxW);
                throw InvalidArg{MB_EINVAL};
            }
            H.nsa.push_back(d->nsa[i]);
            H.nxsa.push_back(d->nxsa[i]);
            H.dx.push_back(d->dx[i]);
            H.gox.push_back(d->gox[i]);
            H.goy.push_back(d->goy[i]);
            H.thetax.push_back(d->thetax[i]);
            H.thetay.push_back(d->thetay[i]);
            H.hs.push_back(d->hs[i]);
            nsa_tot += d->nsa[i];
            H.ngrad += 2L * d->nsa[i];
        }
        std::vector<int> ix(d->sa_ix, d->sa_ix + nsa_tot), iy(d->sa_iy, d->sa_iy + nsa_tot),
            sid(d->sa_stencil, d->sa_stencil + nsa_tot);
        std::vector<long> soff(d->stencil_off, d->stencil_off + d->nstencil);
        // every subaperture's stencil must be one of its WFS's size and inside the table
        long k = 0;
        for (int i = 0; i < d->nwfs; i++) {
            const long len = 2L * (d->nxsa[i] + 2) * (d->nxsa[i] + 2);
            for (int j = 0; j < d->nsa[i]; j++, k++) {
                if (sid[k] < 0 || sid[k] >= d->nstencil || soff[sid[k]] < 0 || soff[sid[k]] + len > d->stencil_len ||
                    ix[k] < 1 || iy[k] < 1) {
                    set_error("mb_geom_wfs_create: subaperture %d of WFS %d: stencil %d or grid index out of range",
                              j, i, sid[k]);
                    throw InvalidArg{MB_EINVAL};
                }
            }
        }
        H.sa_ix.upload(ix);
        H.sa_iy.upload(iy);
        H.sa_st.upload(sid);
        H.st_off.upload(soff);
        std::vector<float> stf(d->stencils, d->stencils + d->stencil_len);
        H.st.upload(stf);
        if (d->nea) {
            std::vector<float> nf(d->nea, d->nea + 3 * nsa_tot);
            H.nea.upload(nf);
            H.have_nea = true;
        }
        for (int l = 0; l < d->natm; l++) {
            if (d->atm_nx[l] < 2 || d->atm_ny[l] < 2 || !(d->atm_dx[l] > 0)) {
                set_error("mb_geom_wfs_create: atmosphere layer %d: %d x %d", l, d->atm_nx[l], d->atm_ny[l]);
                throw InvalidArg{MB_EINVAL};
            }
            // a window must span at most kGeomBlk layer pixels (and fewer than the layer has)
            for (int i = 0; i < d->nwfs; i++) {
                const double sc = std::isfinite(d->hs[i]) ? 1.0 - d->atm_ht[l] / d->hs[i] : 1.0;
                const double step = d->dx[i] * sc / d->atm_dx[l];
                if (!(sc > 0) || step > kGeomMaxStep || kGeomBlk >= d->atm_nx[l] || kGeomBlk >= d->atm_ny[l]) {
                    set_error("mb_geom_wfs_create: layer %d: WFS %d steps %.3g layer pixels per OPD point "
                              "(at most %.3g) on a %d x %d layer", l, i, step, kGeomMaxStep, d->atm_nx[l],
                              d->atm_ny[l]);
                    throw InvalidArg{MB_EUNSUP};
                }
            }
            H.anx.push_back(d->atm_nx[l]);
            H.any.push_back(d->atm_ny[l]);
            H.adx.push_back(d->atm_dx[l]);
            H.aox.push_back(d->atm_ox[l]);
            H.aoy.push_back(d->atm_oy[l]);
            H.aht.push_back(d->atm_ht[l]);
            H.aoff.push_back(H.atm_stride);
            H.atm_stride += (long)d->atm_nx[l] * d->atm_ny[l];
        }
        for (int m = 0; m < d->ndm; m++) {
            if (d->dm_nx[m] < 2 || d->dm_ny[m] < 2 || !(d->dm_dx[m] > 0)) {
                set_error("mb_geom_wfs_create: DM %d: %d x %d", m, d->dm_nx[m], d->dm_ny[m]);
                throw InvalidArg{MB_EINVAL};
            }
            for (int i = 0; i < d->nwfs; i++) {
                const double sc = std::isfinite(d->hs[i]) ? 1.0 - d->dm_ht[m] / d->hs[i] : 1.0;
                const double step = d->dx[i] * sc / d->dm_dx[m];
                if (!(sc > 0) || step > kGeomMaxStep) {
                    set_error("mb_geom_wfs_create: DM %d: WFS %d steps %.3g actuators per OPD point (at most %.3g)",
                              m, i, step, kGeomMaxStep);
                    throw InvalidArg{MB_EUNSUP};
                }
            }
            H.dnx.push_back(d->dm_nx[m]);
            H.dny.push_back(d->dm_ny[m]);
            H.ddx.push_back(d->dm_dx[m]);
            H.dox.push_back(d->dm_ox[m]);
            H.doy.push_back(d->dm_oy[m]);
            H.dht.push_back(d->dm_ht[m]);
            H.doff.push_back(H.nact);
            H.nact += (long)d->dm_nx[m] * d->dm_ny[m];
        }
        H.build_lists(ix, iy, sid, soff, d->stencils);
        H.wind.resize((size_t)H.nbatch * H.natm * 2);
        for (int i = 0; i < H.nbatch; i++)
            for (int l = 0; l < H.natm; l++) {
                H.wind[2 * ((size_t)i * H.natm + l)] = d->atm_vx[l];
                H.wind[2 * ((size_t)i * H.natm + l) + 1] = d->atm_vy[l];
            }
        if (H.natm) H.upload_wind();
        if (H.atm_stride) {
            H.atm.alloc((size_t)H.atm_stride * H.nbatch);
            H.atm.zero_async(nullptr);
        }
        MB_CUDA_TRY(cudaDeviceSynchronize());
    } catch (const CudaError &e) {
        delete h;
        return e.code;
    } catch (const InvalidArg &e) {
        delete h;
        return e.code;
    }
    *out = h;
    return MB_OK;
}

void mb_geom_wfs_free(mb_geom_wfs *h) { delete h; }

long mb_geom_wfs_ngrad(const mb_geom_wfs *h) { return h ? h->H.ngrad : -1; }
long mb_geom_wfs_nact(const mb_geom_wfs *h) { return h ? h->H.nact : -1; }

int mb_geom_wfs_set_atm(mb_geom_wfs *h, int inst, int layer, const double *screen) {
    if (!h || !screen || inst < 0 || inst >= h->H.nbatch || layer < 0 || layer >= h->H.natm) {
        mb::set_error("mb_geom_wfs_set_atm: invalid arguments");
        return MB_EINVAL;
    }
    try {
        mb::GeomWfsHost &H = h->H;
        const long n = (long)H.anx[layer] * H.any[layer];
        std::vector<float> f(screen, screen + n);
        MB_CUDA_TRY(cudaMemcpy(H.atm.p + (size_t)inst * H.atm_stride + H.aoff[layer], f.data(), n * sizeof(float),
                               cudaMemcpyHostToDevice));
    } catch (const mb::CudaError &e) {
        return e.code;
    }
    return MB_OK;
}

int mb_geom_wfs_set_wind(mb_geom_wfs *h, int inst, int layer, double vx, double vy) {
    if (!h || inst < 0 || inst >= h->H.nbatch || layer < 0 || layer >= h->H.natm) {
        mb::set_error("mb_geom_wfs_set_wind: invalid arguments");
        return MB_EINVAL;
    }
    try {
        mb::GeomWfsHost &H = h->H;
        H.wind[2 * ((size_t)inst * H.natm + layer)] = vx;
        H.wind[2 * ((size_t)inst * H.natm + layer) + 1] = vy;
        H.upload_wind();
    } catch (const mb::CudaError &e) {
        return e.code;
    }
    return MB_OK;
}

int mb_geom_wfs_grad(mb_geom_wfs *h, long isim, const float *d_dm, float *d_grad, unsigned long long seed,
                     void *stream) {
    using namespace mb;
    if (!h || !d_grad || isim < 0 || (seed && !h->H.have_nea)) {
        set_error("mb_geom_wfs_grad: invalid arguments%s", h && seed && !h->H.have_nea ? " (no NEA tables)" : "");
        return MB_EINVAL;
    }
    try {
        const GeomWfsHost &H = h->H;
        GeomTab t;
        std::memset(&t, 0, sizeof(t));
        t.nwfs = H.nwfs;
        int ns = 0;
        for (int l = 0; l < H.natm; l++, ns++)
            t.s[ns] = GeomScr{H.atm.p + H.aoff[l], H.atm_stride, H.anx[l], H.any[l], 1.0f, 1};
        if (d_dm)
            for (int m = 0; m < H.ndm; m++, ns++)
                t.s[ns] = GeomScr{d_dm + H.doff[m], H.nact, H.dnx[m], H.dny[m], -1.0f, 0};
        t.nscr = ns;
        t.natm = H.natm;
        for (int i = 0; i < H.nwfs; i++) {
            t.w[i] = H.parts[i];
            for (int s = 0; s < ns; s++) {
                const bool atm = s < H.natm;
                const int q = atm ? s : s - H.natm;
                const double ht = atm ? H.aht[q] : H.dht[q];
                const double sdx = atm ? H.adx[q] : H.ddx[q];
                const double sox = atm ? H.aox[q] : H.dox[q], soy = atm ? H.aoy[q] : H.doy[q];
                const double sc = std::isfinite(H.hs[i]) ? 1.0 - ht / H.hs[i] : 1.0;
                const double dispx = ht * H.thetax[i], dispy = ht * H.thetay[i];
                t.c[i][s] = GeomCoef{H.dx[i] * sc / sdx, (H.gox[i] * sc + dispx - sox) / sdx, H.dx[i] * sc / sdx,
                                     (H.goy[i] * sc + dispy - soy) / sdx};
            }
        }
        const GeomLists L = H.lists();
        if (H.max_blocks) {
            k_wfs_geom<<<dim3((unsigned)H.max_blocks, (unsigned)H.nwfs, (unsigned)H.nbatch), kSepThreads, 0,
                         (cudaStream_t)stream>>>(t, L, H.sa_ix.p, H.sa_iy.p, H.nea.p, H.wind_px.p, d_grad, H.ngrad, isim,
                                                 seed);
            MB_CHECK_LAUNCH();
        }
        if (H.max_dense) {
            const dim3 grid((unsigned)((H.max_dense + kGeomWarps - 1) / kGeomWarps), (unsigned)H.nwfs,
                            (unsigned)H.nbatch);
            k_wfs_dense<<<grid, kGeomWarps * 32, 0, (cudaStream_t)stream>>>(
                t, L, H.sa_ix.p, H.sa_iy.p, H.sa_st.p, H.st.p, H.st_off.p, H.nea.p, H.wind_px.p, d_grad, H.ngrad, isim,
                seed);
            MB_CHECK_LAUNCH();
        }
    } catch (const CudaError &e) {
        return e.code;
    }
    return MB_OK;
}

}  // extern "C"
