// 3D cone-beam separable-footprint projector pair (SF-TR, amplitude A2).
//
// vir's sys_mat/sp.py:93-211 (CTGeometry, footprint1D, forward_project,
// back_project) sketches a separable-footprint cone projector without
// rotation angles.  This is the method it stands in for, the trapezoid /
// rectangle separable footprints of Long, Fessler & Balter, "3D forward and
// back-projection for X-ray CT using separable footprints", IEEE TMI 29(11),
// 2010, on vir's circular cone geometry of dd_fp_cone_3d (sys_mat/dd.py:815):
// source at DSO (cos b, sin b), o = c x + s y, p = -s x + c y,
// u = DSD p / (DSO - o), v = DSD z / (DSO - o); cell edges
// U_j = du (j - nu/2 + su), V_l = dv (l - nv/2 + sv); volume (nx, ny, nz) of
// cubic voxels d; sinogram (na, nu, nv), v fastest.  Voxel (x, y, z) adds
//     f * l_phi0 * l_theta(j, l) * F1(j) * F2(l)
// to cell (j, l), where
//   F1(j): the unit trapezoid through the sorted projections tau0..tau3 of
//          the column's four corners (x +- d/2, y +- d/2), averaged over u cell j;
//   F2(l): the rectangle [M (z - d/2), M (z + d/2)], M = DSD / (DSO - o(x, y)),
//          averaged over v cell l;
//   l_phi0 = d |r| / max(|r_x|, |r_y|), r = (x, y) - DSO (c, s): the path
//          length of the transaxial ray through the column centre;
//   l_theta(j, l) = sqrt(1 + v_l^2 / (u_j^2 + DSD^2)) at the cell centre.
// The forward projection returns these line integrals; the back projection
// is its exact adjoint (vir has no back projector for this footprint).
//
//  FP (sf3d_fp_kernel): warp = 8 u cells x 32-96 v cells of one view; walks the
//    lines and, on each, the columns that cover its cells, see there.
//  BP (sf3d_bp_kernel): the sinogram is first multiplied by l_theta
//    (sf3d_weight, into the workspace, a chunk of views at a time); block =
//    8 x 8 columns x 32 or 64 slices, warp = 8 columns; the two footprints are
//    applied one after the other, see there.
#include <cooperative_groups.h>
#include <math.h>

#include "vg_common.cuh"

namespace {

using namespace vg;
namespace cg = cooperative_groups;

__device__ __forceinline__ float2 view_cs(const double *__restrict__ trig, int ia) {
    return make_float2((float)__ldg(trig + 2 * ia), (float)__ldg(trig + 2 * ia + 1));
}

__device__ __forceinline__ float ucen(const vg_dd3d_geom &g, int j) {
    return g.du * ((float)j + 0.5f - 0.5f * g.nu + g.su);
}
__device__ __forceinline__ float uedge(const vg_dd3d_geom &g, int j) {
    return g.du * ((float)j - 0.5f * g.nu + g.su);
}
__device__ __forceinline__ float vedge(const vg_dd3d_geom &g, int l) {
    return g.dv * ((float)l - 0.5f * g.nv + g.sv);
}
__device__ __forceinline__ float vcen(const vg_dd3d_geom &g, int l) {
    return g.dv * ((float)l + 0.5f - 0.5f * g.nv + g.sv);
}
__device__ __forceinline__ float vox(float d, int i, int n) { return d * ((float)i + 0.5f - 0.5f * n); }

// Footprint of column (x, y): sorted corner projections, l_phi0 and the
// slice height on the detector M d.
struct SfCol {
    float t0, t1, t2, t3, lphi, mz;
};

__device__ __forceinline__ void cswap(float &a, float &b) {
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo;
    b = hi;
}

__device__ __forceinline__ SfCol sf_col(const vg_dd3d_geom &g, float c, float s, float x, float y) {
    const float h = 0.5f * g.d_pix;
    float u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float xx = x + ((q & 1) ? h : -h), yy = y + ((q & 2) ? h : -h);
        const float o = fmaf(c, xx, s * yy), p = fmaf(-s, xx, c * yy);
        u[q] = __fdividef(g.DSD * p, g.DSO - o);
    }
    cswap(u[0], u[1]);
    cswap(u[2], u[3]);
    cswap(u[0], u[2]);
    cswap(u[1], u[3]);
    cswap(u[1], u[2]);
    SfCol C;
    C.t0 = u[0]; C.t1 = u[1]; C.t2 = u[2]; C.t3 = u[3];
    const float rx = x - g.DSO * c, ry = y - g.DSO * s;
    C.lphi = __fdividef(g.d_pix * sqrtf(rx * rx + ry * ry), fmaxf(fabsf(rx), fabsf(ry)));
    C.mz = __fdividef(g.DSD * g.d_pix, g.DSO - fmaf(c, x, s * y));
    return C;
}

// Integral of the unit trapezoid (t0, t1, t2, t3) from -inf to u: the parts of
// the rise, the top and the fall before u (no branches: lanes hold footprints
// at all stages).
__device__ __forceinline__ float trap_cum(float u, const SfCol &C) {
    const float a = fminf(fmaxf(u, C.t0), C.t1) - C.t0, b = fminf(fmaxf(u, C.t1), C.t2) - C.t1;
    const float f = C.t3 - C.t2, e = C.t3 - fminf(fmaxf(u, C.t2), C.t3);
    const float rise = __fdividef(a * a, fmaxf(2.f * (C.t1 - C.t0), 1e-30f));
    const float fall = 0.5f * f - __fdividef(e * e, fmaxf(2.f * f, 1e-30f));
    return rise + b + fall;
}

// F1 averaged over [ua, ub] (cell width du), times l_phi0
__device__ __forceinline__ float uweight(const SfCol &C, float ua, float ub, float inv_du) {
    return (trap_cum(ub, C) - trap_cum(ua, C)) * inv_du * C.lphi;
}

// Fractional pixel index, along the driving axis, of the point of the line
// at orthogonal coordinate `cen` that projects to u (x, y = (b, cen) when
// X-driven, else (cen, b)):  b (DSD pd + u od) = u (DSO - oc) - DSD pc.
__device__ __forceinline__ float unproj_idx(const vg_dd3d_geom &g, float c, float s, bool xdrv,
                                            float cen, float u, int nd) {
    const float pd = xdrv ? -s : c, od = xdrv ? c : s;
    const float pc = xdrv ? c * cen : -s * cen, oc = xdrv ? s * cen : c * cen;
    const float b = __fdividef(u * (g.DSO - oc) - g.DSD * pc, g.DSD * pd + u * od);
    return __fdividef(b, g.d_pix) + 0.5f * nd;
}

// ---------------------------------------------------------------------------
// Forward projection
// ---------------------------------------------------------------------------
// A warp owns 8 u cells x 32 M v cells of one view and walks the orthogonal
// lines of the volume.  The ranges of columns that reach its u cells are found
// 32 lines at a time (lane = line), a line's footprints, F1 l_phi0 weights on
// the 8 cells and v maps 32 columns at a time (lane = column).  Then per column
// that covers any of the cells: its slices under the tile's v cells go to shared
// memory (one 16-byte load per 4 slices, the next column's issued before this
// one is used), every lane sums its M v cells' 2-5 slices with their overlaps,
// and adds the result to the cells the column covers.  Overlaps are counted in
// slices from the tile's middle.  LONG: v cells over more slices than a row buffer
// holds; every lane takes its cells' sums from running sums of the column (128^3, 180
// views, v cells of 4, 6 and 10 slices: 1.5, 0.97 and 0.97 ms; cell by cell from the
// volume 9.1, 9.6 and 11.4; the slices through the row buffer 3.1, 1.9 and 2.0).  Sums:
// 16 lines in registers, then a second running sum in shared memory.
//
// Bound by instruction issue (66 %, 213 per column and line for 8 x 96 cells).
// 256^3, 360 views of 512 x 384: 55.3 -> 21.6 ms against profiles of every column
// in block-wide tables, one barrier per line (144 instructions per 32 cells and
// line); the weights by branches per lane and the FMAs by cell 28 ms.  4 blocks
// per SM 21.6, 5 22.5, 6 22.4 ms.
constexpr int SFW = 4, SF_FP_MINB = 4, SF_LONG_MINB = 6;  // warps per block
constexpr int UC = 8;                   // u cells per warp
constexpr int BW = 128;                 // entries of a row buffer

// The entries of a column's zn outputs, B each, the middle one (zn / 2) at entry
// ci + t of the input (t the product with B, ci + cf the offset): they are counted
// from c = floor(t) + ci, so an output carries the rounding of its distance from the
// middle; the window that is staged starts at or below the first output's entry,
// found with the v step's expression.
struct Win {
    float y;               // the middle output from c on
    int start, mid, rows;  // c - start, entries of the window
};
template <int VEC>
__device__ __forceinline__ Win win_at(float B, float t, float cf, float ci, int zn) {
    Win w;
    const float tf = floorf(t), lo = -(float)(zn >> 1), u = fminf(t - tf, 0.99999994f) + cf, uf = floorf(u);
    const int c = (int)tf + (int)ci + (int)uf;
    w.y = u - uf;  // below 1, so that the start is at c at most
    w.start = c + __float2int_rd(fmaf(B, lo, w.y));
    if (VEC == 4) w.start &= ~3;
    w.mid = c - w.start;
    w.rows = w.mid + __float2int_rd(fmaf(B, (float)zn + lo, w.y)) + 1;
    return w;
}

struct SfFpWarp {
    float T[2][BW];
    float w[32][UC];  // per column: F1 l_phi0 M d / dv on the u cells
    float4 rec[32];   // slices per v cell, Win's y and start, index of the column
    int mr[32];       // Win's mid | rows << 12
};

// LONG: running sums of the volume's columns over z, from 0 again every 1 << lz slices
// (from the volume's start they would carry the rounding of the column's total).
__global__ void __launch_bounds__(256)
sf3d_zsums(vg_dd3d_geom g, const float *__restrict__ vol, int lz, float *__restrict__ zs) {
    const int lane = threadIdx.x & 31, per = (g.nz + 31) >> 5;
    const size_t n = (size_t)g.nx * g.ny * per;
    for (size_t w = ((size_t)blockIdx.x * 256 + threadIdx.x) >> 5; w < n; w += (size_t)gridDim.x * 8) {
        const size_t col = w / per;
        const int z = (int)(w - col * per) * 32 + lane;
        float v = z < g.nz ? __ldg(vol + col * g.nz + z) : 0.f;
        for (int o = 1; o < 1 << lz; o <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, v, o);
            if ((lane & ((1 << lz) - 1)) >= o) v += t;
        }
        if (z < g.nz) zs[col * g.nz + z] = v;
    }
}

// LONG: a v cell from position tl to th, in slices from the c-th on: a part of its first
// slice, those between, a part of its last.  f: the column, L: its running sums.
__device__ __forceinline__ float long_cell(const float *f, const float *L, int nz, int lz, int c, float B, float tl,
                                           float th) {
    tl = fminf(fmaxf(tl, -1073741824.f), 1073741824.f);  // the rows below are int
    th = fminf(fmaxf(th, -1073741824.f), 1073741824.f);
    const float fl = floorf(tl), fh = floorf(th), w0 = fminf(B, (fl + 1.0f) - tl), w1 = fh > fl ? th - fh : 0.f;
    const int r0 = c + (int)fl, r1 = c + (int)fh;
    const int lo = max(r0 + 1, 0), hi = min(r1, nz);  // whole slices lo .. hi - 1
    const bool whole = hi > lo;
    const int b0 = lo >> lz, b1 = whole ? (hi - 1) >> lz : b0;
    const float end = whole ? __ldg(L + hi - 1) : 0.f;
    const float before = whole && (lo & ((1 << lz) - 1)) ? __ldg(L + lo - 1) : 0.f;
    const float first = b0 < b1 ? __ldg(L + ((b0 + 1) << lz) - 1) : 0.f;
    const float f0 = (unsigned)r0 < (unsigned)nz ? __ldg(f + r0) : 0.f;
    const float f1 = w1 > 0.f && (unsigned)r1 < (unsigned)nz ? __ldg(f + r1) : 0.f;
    float s = (first - before) + end;
    for (int b = b0 + 1; b < b1; ++b) s += __ldg(L + ((b + 1) << lz) - 1);
    s = fmaf(w0, f0, fmaf(w1, f1, s));
    if (!(fabsf(s) < INFINITY)) {  // the running sums take infinities and NaN past their slice
        s = 0.f;
        for (int z = lo; z < hi; ++z) s += __ldg(f + z);
        if ((unsigned)r0 < (unsigned)nz) s = fmaf(w0, __ldg(f + r0), s);
        if (w1 > 0.f && (unsigned)r1 < (unsigned)nz) s = fmaf(w1, __ldg(f + r1), s);
    }
    return s;
}

template <int VEC, int M, bool LONG>
__global__ void __launch_bounds__(32 * SFW, LONG ? SF_LONG_MINB : SF_FP_MINB)
sf3d_fp_kernel(vg_dd3d_geom g, const float *__restrict__ vol, const double *__restrict__ trig,
               float *__restrict__ sino, const float *__restrict__ zs, int lz) {
    constexpr int SZ = 32 * M, NW = M >= 2 ? 3 : 5;
    extern __shared__ float4 smem4[];
    const int ia = blockIdx.z, v0 = blockIdx.x * SZ;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = (blockIdx.y * SFW + warp) * UC;
    SfFpWarp &W = reinterpret_cast<SfFpWarp *>(smem4)[warp];
    float *acc = reinterpret_cast<float *>(reinterpret_cast<SfFpWarp *>(smem4) + SFW) + warp * UC * SZ + lane;
    if (u0 >= g.nu) return;  // no block barriers below
    const float2 cs = view_cs(trig, ia);
    const float c = cs.x, s = cs.y;
    const bool xdrv = fabsf(s) >= fabsf(c);
    const int nd = xdrv ? g.nx : g.ny, no = xdrv ? g.ny : g.nx;
    const float inv_du = 1.0f / g.du;
    const int nuT = min(UC, g.nu - u0), zn = min(SZ, g.nv - v0);
    const float TUa = uedge(g, u0), TUb = uedge(g, u0 + nuT);
    // the inverse edge map has a pole at u = -DSD pd / od; cells holding it (or
    // within two cells of it) cannot bound their columns through the map
    const float pd = xdrv ? -s : c, od = xdrv ? c : s;
    bool pole = false;
    if (od != 0.f) {
        const float up = -g.DSD * pd / od;
        pole = up >= TUa - 2.f * g.du && up <= TUb + 2.f * g.du;
    }
    const float kB = g.dv / (g.DSD * g.d_pix);  // slices per v cell = kB (DSO - o)
    const float vd = (float)(v0 + (zn >> 1)) - 0.5f * g.nv + g.sv;  // the middle v cell's edge
    const float ci = floorf(0.5f * g.nz), cf = 0.5f * g.nz - ci;
    float2 grp[UC / 2][M];  // u cells in pairs
#pragma unroll
    for (int q = 0; q < UC; ++q)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            grp[q / 2][m] = dup(0.f);
            acc[q * SZ + 32 * m] = 0.f;
        }
    // a column's profile p at this lane's v cells to the 8 u cells (odd: not finite in some
    // lane)
    auto spread = [&](const float (&p)[M], bool odd, float4 wa, float4 wb) {
        const float2 w2[UC / 2] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w),
                                   make_float2(wb.x, wb.y), make_float2(wb.z, wb.w)};
        if (!odd) {
#pragma unroll
            for (int q = 0; q < UC / 2; ++q)
#pragma unroll
                for (int m = 0; m < M; ++m) grp[q][m] = pk_fma(w2[q], dup(p[m]), grp[q][m]);
        } else {  // infinities and NaN only to the cells that the column covers
#pragma unroll
            for (int q = 0; q < UC / 2; ++q)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    if (w2[q].x != 0.f) grp[q][m].x = fmaf(w2[q].x, p[m], grp[q][m].x);
                    if (w2[q].y != 0.f) grp[q][m].y = fmaf(w2[q].y, p[m], grp[q][m].y);
                }
        }
    };
    int ngrp = 0;
    for (int lb = 0; lb < no; lb += 32) {
        // columns of line lb + lane whose footprints can reach the cells: the map of
        // their outer edges (widened by a cell) on both boundaries of the line, one
        // column of margin each side
        int kA = 0, kE = -1;
        if (lb + lane < no) {
            kE = nd - 1;
            if (!pole) {
                const float cj = vox(g.d_pix, lb + lane, no), h = 0.5f * g.d_pix;
                const float a0 = unproj_idx(g, c, s, xdrv, cj - h, TUa - g.du, nd);
                const float a1 = unproj_idx(g, c, s, xdrv, cj + h, TUa - g.du, nd);
                const float b0 = unproj_idx(g, c, s, xdrv, cj - h, TUb + g.du, nd);
                const float b1 = unproj_idx(g, c, s, xdrv, cj + h, TUb + g.du, nd);
                const float lo = fminf(fminf(a0, a1), fminf(b0, b1));
                const float hi = fmaxf(fmaxf(a0, a1), fmaxf(b0, b1));
                kA = max((int)floorf(fmaxf(lo, -2.f)) - 1, 0);
                kE = min((int)floorf(fminf(hi, (float)nd + 2.f)) + 1, nd - 1);
            }
        }
        unsigned lines = __ballot_sync(0xffffffffu, kE >= kA);
        while (lines) {
            const int l = __ffs(lines) - 1, io = lb + l;
            lines &= lines - 1;
            const int ka = __shfl_sync(0xffffffffu, kA, l), ke = __shfl_sync(0xffffffffu, kE, l);
            bool some = false;
            for (int kc = ka; kc <= ke; kc += 32) {  // 32 columns of the line at a time
                // this lane's column
                float w[UC];
                float B = 1.f;
                Win wn = {};
                int cidx = 0;
                bool any = false;
                if (kc + lane <= ke) {
                    const int k = kc + lane;
                    const float cen = vox(g.d_pix, io, no), bx = vox(g.d_pix, k, nd);
                    const float x = xdrv ? bx : cen, y = xdrv ? cen : bx;
                    const SfCol C = sf_col(g, c, s, x, y);
                    if (C.t3 > TUa && C.t0 < TUb) {
                        const float f = inv_du * C.lphi * C.mz / g.dv;
                        float e = trap_cum(TUa, C);
#pragma unroll
                        for (int q = 0; q < UC; ++q) {
                            const float t = trap_cum(uedge(g, u0 + q + 1), C);
                            w[q] = q < nuT ? (t - e) * f : 0.f;
                            any |= w[q] != 0.f;
                            e = t;
                        }
                        B = kB * (g.DSO - fmaf(c, x, s * y));
                        wn = win_at<VEC>(B, B * vd, cf, ci, zn);
                        if (!LONG && (wn.start + wn.rows <= 0 || wn.start >= g.nz)) any = false;
                        cidx = xdrv ? k * g.ny + io : io * g.ny + k;
                    }
                }
                unsigned cols = __ballot_sync(0xffffffffu, any);
                if (!cols) continue;
                some = true;
                if (any) {
                    *reinterpret_cast<float4 *>(&W.w[lane][0]) = make_float4(w[0], w[1], w[2], w[3]);
                    *reinterpret_cast<float4 *>(&W.w[lane][4]) = make_float4(w[4], w[5], w[6], w[7]);
                    W.rec[lane] = make_float4(B, wn.y, __int_as_float(LONG ? wn.start + wn.mid : wn.start),
                                              __int_as_float(cidx));
                    W.mr[lane] = wn.mid | wn.rows << 12;
                }
                __syncwarp();
                if (LONG) {
                    for (; cols; cols &= cols - 1) {
                        const int t = __ffs(cols) - 1;
                        const float4 rc = W.rec[t];
                        const int mid = max(min(__float_as_int(rc.z), 1 << 29), -(1 << 29));
                        const size_t o = (size_t)__float_as_uint(rc.w) * g.nz;
                        float p[M];
                        bool odd = false;
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            const float vm = (float)(min(32 * m + lane, zn - 1) - (zn >> 1));
                            p[m] = long_cell(vol + o, zs + o, g.nz, lz, mid, rc.x, fmaf(rc.x, vm, rc.y),
                                             fmaf(rc.x, vm + 1.0f, rc.y));
                            odd |= !(fabsf(p[m]) < INFINITY);
                        }
                        spread(p, __any_sync(0xffffffffu, odd), *reinterpret_cast<const float4 *>(&W.w[t][0]),
                               *reinterpret_cast<const float4 *>(&W.w[t][4]));
                    }
                    __syncwarp();  // the table is reused
                    continue;
                }
                int win = 0;
                float2 r[2];
                float4 rc;
                int mr;
                unsigned in = 0;
                auto load = [&](int t) {  // column t's slices that this lane loads, clamped to the volume
                    rc = W.rec[t];
                    mr = W.mr[t];
                    const int zs = __float_as_int(rc.z);
                    win = (mr >> 12) + NW - 1;
                    const char *p = ptr_at(reinterpret_cast<const char *>(vol), __float_as_int(rc.w), 4u * g.nz);
                    in = 0;
                    auto at = [&](int i) {
                        const int z = zs + min(VEC == 4 ? 4 * lane : lane + 32 * i, (win - 1) & ~(VEC - 1));
                        const int zc = min(max(z, 0), g.nz - VEC);
                        in |= (unsigned)(zc == z) << i;
                        return p + 4 * zc;
                    };
                    if (VEC == 4) {
                        const float4 f = __ldg(reinterpret_cast<const float4 *>(at(0)));
                        r[0] = make_float2(f.x, f.y);
                        r[1] = make_float2(f.z, f.w);
                    } else {
                        r[0] = make_float2(__ldg(reinterpret_cast<const float *>(at(0))),
                                           __ldg(reinterpret_cast<const float *>(at(1))));
                        if (win > 64)
                            r[1] = make_float2(__ldg(reinterpret_cast<const float *>(at(2))),
                                               __ldg(reinterpret_cast<const float *>(at(3))));
                    }
                };
                int t = __ffs(cols) - 1, buf = 0;
                load(t);
                for (;;) {
                    float *T = W.T[buf];
                    buf ^= 1;
                    // slices outside the volume count as 0
                    if (VEC == 4) {
                        if (4 * lane < win)
                            *reinterpret_cast<float4 *>(T + 4 * lane) =
                                in ? make_float4(r[0].x, r[0].y, r[1].x, r[1].y) : make_float4(0.f, 0.f, 0.f, 0.f);
                    } else {
                        T[lane] = in & 1 ? r[0].x : 0.f;
                        T[lane + 32] = in & 2 ? r[0].y : 0.f;
                        if (win > 64) {
                            T[lane + 64] = in & 4 ? r[1].x : 0.f;
                            T[lane + 96] = in & 8 ? r[1].y : 0.f;
                        }
                    }
                    __syncwarp();
                    const float4 cur = rc;
                    const int mid = mr & 0xfff;
                    const float4 wa = *reinterpret_cast<const float4 *>(&W.w[t][0]);
                    const float4 wb = *reinterpret_cast<const float4 *>(&W.w[t][4]);
                    cols &= cols - 1;
                    if (cols) {
                        t = __ffs(cols) - 1;
                        load(t);
                    }
                    // this column's profile at the lane's v cells
                    float p[M];
                    bool odd = false;
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const float vm = (float)(32 * m + lane - (zn >> 1));
                        const float tl = fmaf(cur.x, vm, cur.y), th = fmaf(cur.x, vm + 1.0f, cur.y);
                        const float tf = floorf(tl);
                        const float *q = T + min((int)tf + mid, BW - NW);  // v cells past the detector read anything
                        float a = (fminf(th, tf + 1.0f) - tl) * q[0];
                        a = fmaf(__saturatef(th - (tf + 1.0f)), q[1], a);
#pragma unroll
                        for (int i = 2; i < NW; ++i) {
                            const float wi = __saturatef(th - (tf + (float)i));
                            a = fmaf(wi, lds_if(q + i, wi), a);
                        }
                        p[m] = a;
                        odd |= !(fabsf(a) < INFINITY);
                    }
                    odd = __any_sync(0xffffffffu, odd);
                    if (odd) {  // infinities and NaN only to the v cells that overlap them
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            const float vm = (float)(32 * m + lane - (zn >> 1));
                            const float tl = fmaf(cur.x, vm, cur.y), th = fmaf(cur.x, vm + 1.0f, cur.y);
                            const float tf = floorf(tl);
                            const float *q = T + min((int)tf + mid, BW - NW);
                            p[m] = 0.f;
                            for (int i = 0; i < NW; ++i) {
                                const float wi = fminf(th, tf + (float)(i + 1)) - fmaxf(tl, tf + (float)i);
                                if (wi > 0.f) p[m] = fmaf(wi, q[i], p[m]);
                            }
                        }
                    }
                    spread(p, odd, wa, wb);
                    if (!cols) break;
                }
                __syncwarp();  // the table and the row buffers are reused
            }
            if (!some) continue;
            if (++ngrp == 16) {
#pragma unroll
                for (int q = 0; q < UC; ++q)
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        acc[q * SZ + 32 * m] += q & 1 ? grp[q / 2][m].y : grp[q / 2][m].x;
                        if (q & 1) grp[q / 2][m] = dup(0.f);
                    }
                ngrp = 0;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < UC; ++q)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int j = u0 + q, l = v0 + 32 * m + lane;
            if (j < g.nu && l < g.nv) {
                const float uc = ucen(g, j), vc = vcen(g, l);
                const float lth = sqrtf(1.f + vc * vc / (uc * uc + g.DSD * g.DSD));
                sino[((size_t)ia * g.nu + j) * g.nv + l] = 
                    (acc[q * SZ + 32 * m] + (q & 1 ? grp[q / 2][m].y : grp[q / 2][m].x)) * lth;
            }
        }
}

template <int VEC, int M, bool LONG = false>
int launch_fp(const vg_dd3d_geom *g, const float *vol, const double *trig, float *sino, cudaStream_t st,
              const float *zs = nullptr, int lz = 0) {
    constexpr size_t smem = SFW * (sizeof(SfFpWarp) + UC * 32 * M * sizeof(float));
    int s = cuda_status(cudaFuncSetAttribute(sf3d_fp_kernel<VEC, M, LONG>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "sf3d_fp");
    if (s) return s;
    dim3 grid(ceil_div(g->nv, 32 * M), ceil_div(g->nu, UC * SFW), g->na);
    sf3d_fp_kernel<VEC, M, LONG><<<grid, 32 * SFW, smem, st>>>(*g, vol, trig, sino, zs, lz);
    return launch_status("sf3d_fp");
}

// ---------------------------------------------------------------------------
// Back projection
// ---------------------------------------------------------------------------

// out[a - a0] = sino[a] * l_theta, views a0 .. a0 + cnt - 1
__global__ void sf3d_weight(vg_dd3d_geom g, const float *__restrict__ sino, int a0, int cnt,
                            float *__restrict__ out) {
    const size_t n = (size_t)cnt * g.nu * g.nv;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const int l = (int)(i % g.nv);
        const int j = (int)((i / g.nv) % g.nu);
        const float uc = ucen(g, j), vc = vcen(g, l);
        const float lth = sqrtf(1.f + vc * vc / (uc * uc + g.DSD * g.DSD));
        out[i] = sino[(size_t)a0 * g.nu * g.nv + i] * lth;
    }
}

// The footprints are applied one after the other.  A warp owns 8 columns and
// 32 M slices of each, and walks the views, 4 at a time (their F1 l_phi0 weights
// and v maps tabulated at once, lane = view x column).  Per column and view it
//   u: adds the 1-4 u cells under the column, times F1 l_phi0, over the window of
//      v cells its slices project to (16-byte loads, lane = 4 cells), into a row
//      buffer in shared memory;
//   v: lets every slice add its 2-5 cells of the buffer with their overlaps.
// Overlaps are in cell units, counted from the tile's middle.  Sums: 16
// views in registers, then a compensated sum per voxel in shared memory.
// Columns over more than 4 u cells, or whose slices reach more cells than the
// buffer holds, few here, take a per-voxel path.  With too few tiles to fill the GPU the
// blocks of a cluster share a tile's views; sums meet in rank order.
//
// 256^3, 360 views of 512 x 384: 43.0 -> 16.6 ms (62 instructions per 32 voxels and
// view against 228, bound by issue and the latency of the loads; 2 blocks per SM
// 18.1 ms).  With 4-byte loads, or 32 slices, the 80 registers of 3 blocks spill: 2 there
// (128 x 128 x 97, 180 views: 1.62 -> 1.52 ms).
constexpr int BT = 8, BKU = 4;
constexpr int BP_GROUP = 16;

struct SfBpWarp {
    float T[2][2][BW];
    float4 w[4][BT];    // F1 l_phi0 / dv of u cells j0 .. j0 + 3
    float4 rec[4][BT];  // v cells per slice, Win's y and start, j0 | count << 21
    int mr[4][BT];      // Win's mid | rows << 12
};

// one voxel, one view, straight from the weighted sinogram (any geometry)
__device__ __noinline__ float sf_voxel_view(const vg_dd3d_geom &g, const float *__restrict__ q,
                                            float c, float s, float x, float y, int iz) {
    const SfCol C = sf_col(g, c, s, x, y);
    const float inv_du = 1.0f / g.du, inv_dv = 1.0f / g.dv;
    const float U0 = uedge(g, 0), V0 = vedge(g, 0);
    const int ja = max((int)floorf((C.t0 - U0) * inv_du), 0);
    const int jb = min((int)floorf((C.t3 - U0) * inv_du), g.nu - 1);
    const float va = C.mz * ((float)iz - 0.5f * g.nz), vb = va + C.mz;
    const int la = max((int)floorf((va - V0) * inv_dv), 0);
    const int lb = min((int)floorf((vb - V0) * inv_dv), g.nv - 1);
    float part = 0.f;
    for (int j = ja; j <= jb; ++j) {
        const float w = uweight(C, uedge(g, j), uedge(g, j + 1), inv_du);
        if (w == 0.f) continue;
        float r = 0.f;
        for (int l = la; l <= lb; ++l) {
            const float ov = fminf(vb, vedge(g, l + 1)) - fmaxf(va, vedge(g, l));
            if (ov > 0.f) r = fmaf(__ldg(q + (size_t)j * g.nv + l), ov, r);
        }
        part = fmaf(w, r, part);
    }
    return part * inv_dv;
}

// views [ia, ie) of 8 columns (x0 + c, iy) and the slices z0 + lane + 32 i < z0 + sz,
// voxel by voxel, added to their sums at kh
__device__ __noinline__ void sf_views_again(const vg_dd3d_geom &g, const float *__restrict__ qw,
                                            const double *__restrict__ trig, int a0, int ia, int ie, int x0, int iy,
                                            int z0, int sz, float2 *kh) {
    for (int c = 0; c < BT && x0 + c < g.nx && iy < g.ny; ++c)
        for (int z = threadIdx.x & 31; z < sz && z0 + z < g.nz; z += 32) {
            float t = 0.f;
            for (int a = ia; a < ie; ++a) {
                const float2 cs = view_cs(trig, a0 + a);
                t += sf_voxel_view(g, qw + (size_t)a * g.nu * g.nv, cs.x, cs.y, vox(g.d_pix, x0 + c, g.nx),
                                   vox(g.d_pix, iy, g.ny), z0 + z);
            }
            Kahan k;
            k.s = kh[c * sz + z].x; k.c = kh[c * sz + z].y;
            k.add(t);
            kh[c * sz + z] = make_float2(k.s, k.c);
        }
}

constexpr int SF_BP_MINB = 3, SF_WIDE_MINB = 3;

template <int VEC, int M>
__global__ void __launch_bounds__(256, VEC == 1 || M == 1 ? 2 : SF_BP_MINB)
sf3d_bp_kernel(vg_dd3d_geom g, const float *__restrict__ qw, const double *__restrict__ trig, int a0,
               int cnt, int accumulate, float *__restrict__ vol) {
    constexpr int SZ = 32 * M, NW = M == 2 ? 3 : 5, NV = 4 / VEC;
    extern __shared__ float4 smem4[];
    float2 *kh = reinterpret_cast<float2 *>(smem4);  // [BT * BT][SZ] (sum, compensation)
    cg::cluster_group cl = cg::this_cluster();
    const int S = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int z0 = (blockIdx.x / S) * SZ, y0 = blockIdx.y * BT, x0 = blockIdx.z * BT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    SfBpWarp &W = reinterpret_cast<SfBpWarp *>(kh + BT * BT * SZ)[warp];
    const int iy = y0 + warp, zn = min(SZ, g.nz - z0);
    const float inv_du = 1.0f / g.du, U0 = uedge(g, 0);
    const float zd = (float)(z0 + (zn >> 1)) - 0.5f * g.nz;  // the middle slice's edge, exact
    const float cv = 0.5f * g.nv - g.sv, ci = floorf(cv), cf = cv - ci;  // cell coordinate of v = 0
    const float zl = (float)(lane - (zn >> 1));
    for (int c = warp; c < BT * BT; c += 8)
        for (int m = 0; m < M; ++m) kh[c * SZ + 32 * m + lane] = make_float2(0.f, 0.f);
    __syncthreads();
    float grp[BT][M];
#pragma unroll
    for (int c = 0; c < BT; ++c)
#pragma unroll
        for (int m = 0; m < M; ++m) grp[c][m] = 0.f;
    int ngrp = 0;
    // the sums of the ngrp views before view ie
    auto flush = [&](int ie) {
        bool odd = false;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            float t = grp[0][m];
#pragma unroll
            for (int c = 1; c < BT; ++c) t += grp[c][m];
            odd |= 32 * m + lane < zn && !(fabsf(t) < INFINITY);
        }
        // infinities and NaN only to the slices that their cells overlap: the v step
        // multiplies cells of weight 0 too, so these views again, voxel by voxel
        if (__any_sync(0xffffffffu, odd)) {
            sf_views_again(g, qw, trig, a0, ie - ngrp, ie, x0, iy, z0, SZ, kh + BT * warp * SZ);
        } else {
#pragma unroll
            for (int c = 0; c < BT; ++c)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    float2 *k = kh + (c + BT * warp) * SZ + 32 * m + lane;
                    Kahan a;
                    a.s = k->x; a.c = k->y;
                    a.add(grp[c][m]);
                    *k = make_float2(a.s, a.c);
                }
        }
#pragma unroll
        for (int c = 0; c < BT; ++c)
#pragma unroll
            for (int m = 0; m < M; ++m) grp[c][m] = 0.f;
        ngrp = 0;
    };
    const int va0 = (int)((long long)cnt * rank / S), va1 = (int)((long long)cnt * (rank + 1) / S);
    for (int ib = va0; ib < va1; ib += 4) {
        unsigned slow, live;
        {
            const int sv = lane >> 3, c = lane & 7, ix = x0 + c;
            const float2 cs = view_cs(trig, a0 + min(ib + sv, cnt - 1));
            float w[BKU] = {0.f, 0.f, 0.f, 0.f};
            float B = 1.f;
            Win r = {};
            int j0 = 0, n = 0;
            bool far = false;
            if (ix < g.nx && iy < g.ny) {
                const SfCol C = sf_col(g, cs.x, cs.y, vox(g.d_pix, ix, g.nx), vox(g.d_pix, iy, g.ny));
                const int ja = (int)floorf((C.t0 - U0) * inv_du), jb = (int)floorf((C.t3 - U0) * inv_du);
                j0 = min(max(ja, 0), g.nu - 1);
                n = max(min(jb, g.nu - 1) - max(ja, 0) + 1, 0);
                if (jb - ja >= BKU) n = n > 0 ? BKU + 1 : 0;
                float e = trap_cum(uedge(g, j0), C);
                const float f = inv_du * C.lphi;
#pragma unroll
                for (int t = 0; t < BKU; ++t) {
                    const float h = trap_cum(uedge(g, j0 + t + 1), C);
                    w[t] = t < n ? (h - e) * f : 0.f;
                    e = h;
                }
                B = C.mz / g.dv;
                r = win_at<VEC>(B, B * zd, cf, ci, zn);
                far = r.start + r.rows <= 0 || r.start >= g.nv;
                if (B > NW - 1.0f || r.rows > BW - NW + 1) n = n > 0 ? BKU + 1 : 0;
            }
            if (far) n = 0;
            slow = __ballot_sync(0xffffffffu, n > BKU);
            live = __ballot_sync(0xffffffffu, n > 0);
            W.w[sv][c] = make_float4(w[0], w[1], w[2], w[3]);
            W.rec[sv][c] = make_float4(B, r.y, __int_as_float(r.start), __int_as_float(j0 | n << 21));
            W.mr[sv][c] = r.mid | r.rows << 12;
            __syncwarp();
        }
        const int nb = min(4, va1 - ib);
        for (int sv = 0; sv < nb; ++sv) {
            const unsigned lv = live >> (8 * sv) & 0xff, sl = slow >> (8 * sv) & 0xff;
            const char *q = reinterpret_cast<const char *>(qw + (size_t)(ib + sv) * g.nu * g.nv);
#pragma unroll
            for (int c0 = 0; c0 < BT; c0 += 2) {
                // every pair has a barrier, also one that uses no row buffer: it lies
                // between the reads of the pair before and the next stores there
                if (!(lv >> c0 & 3)) {
                    __syncwarp();
                    continue;
                }
                if (sl >> c0 & 3) {
                    const float2 cs = view_cs(trig, a0 + ib + sv);
#pragma unroll
                    for (int c = c0; c < c0 + 2; ++c)
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            const int iz = z0 + 32 * m + lane;
                            if (x0 + c < g.nx && iz < g.nz)
                                grp[c][m] += sf_voxel_view(g, reinterpret_cast<const float *>(q), cs.x, cs.y,
                                                           vox(g.d_pix, x0 + c, g.nx),
                                                           vox(g.d_pix, iy, g.ny), iz);
                        }
                    __syncwarp();
                    continue;
                }
                float (*T)[BW] = W.T[c0 >> 1 & 1];
                float wv[2][M][NW];
                int qi[2][M];
                bool two[2];
                float2 o[2][2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 w = W.w[sv][c0 + h], rc = W.rec[sv][c0 + h];
                    const int vs = __float_as_int(rc.z);
                    const int bits = __float_as_int(rc.w), n = bits >> 21, mr = W.mr[sv][c0 + h], mid = mr & 0xfff;
                    const unsigned j = bits & 0x1fffff;  // nu < 2^21
                    const int win = (mr >> 12) + NW - 1;
                    // this lane's cells, clamped to the window and the detector
                    int vo[NV];
                    unsigned in = 0;
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        const int v = vs + min(VEC == 4 ? 4 * lane : lane + 32 * i, (win - 1) & ~(VEC - 1));
                        vo[i] = 4 * min(max(v, 0), g.nv - VEC);
                        in |= (unsigned)(vo[i] == 4 * v) << i;
                    }
                    const char *p = VEC == 4 ? q + vo[0] : q;
                    auto load = [&](unsigned jj, float2 (&r)[2]) {
                        const char *a = ptr_at(p, jj, 4u * g.nv);
                        if (VEC == 4) {
                            const float4 f = __ldg(reinterpret_cast<const float4 *>(a));
                            r[0] = make_float2(f.x, f.y);
                            r[1] = make_float2(f.z, f.w);
                        } else {
                            auto at = [&](int i) {
                                return __ldg(reinterpret_cast<const float *>(a + vo[i & (NV - 1)]));
                            };
                            r[0] = make_float2(at(0), at(1));
                            if (win > 64) r[1] = make_float2(at(2), at(3));
                        }
                    };
                    float2 r0[2], r1[2], r2[2];
                    load(j, r0);
                    load(j + (n > 1), r1);
                    load(j + (n > 2 ? 2 : n > 1 ? 1 : 0), r2);
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        o[h][i] = pk_fma(dup(w.z), r2[i], pk_fma(dup(w.y), r1[i], pk_mul(dup(w.x), r0[i])));
                    if (n > 3) {
                        load(j + 3, r0);
#pragma unroll
                        for (int i = 0; i < 2; ++i) o[h][i] = pk_fma(dup(w.w), r0[i], o[h][i]);
                    }
                    // nothing from the nearest u cell of a column beside the detector, and from
                    // v cells outside it
                    if (n == 0) in = 0;
                    if (VEC == 4) {
                        if (!in) o[h][0] = o[h][1] = dup(0.f);
                    } else {
                        if (!(in & 1)) o[h][0].x = 0.f;
                        if (!(in & 2)) o[h][0].y = 0.f;
                        if (!(in & 4)) o[h][1].x = 0.f;
                        if (!(in & 8)) o[h][1].y = 0.f;
                    }
                    // overlaps of this lane's slices with their cells
                    float over = 0.f;
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const float zm = zl + (float)(32 * m);
                        const float tl = fmaf(rc.x, zm, rc.y), th = fmaf(rc.x, zm + 1.0f, rc.y);
                        const float tf = floorf(tl);
                        wv[h][m][0] = fminf(th, tf + 1.0f) - tl;
#pragma unroll
                        for (int t = 1; t < NW; ++t) wv[h][m][t] = __saturatef(th - (tf + (float)t));
                        if (32 * m + lane < zn) over = fmaxf(over, th - tf);
                        qi[h][m] = min((int)tf + mid, BW - NW);  // slices past the volume read anything
                    }
                    two[h] = !__any_sync(0xffffffffu, over > 2.0f);
                    if (VEC == 4) {
                        if (4 * lane < win)
                            *reinterpret_cast<float4 *>(T[h] + 4 * lane) =
                                make_float4(o[h][0].x, o[h][0].y, o[h][1].x, o[h][1].y);
                    } else {
                        T[h][lane] = o[h][0].x;
                        T[h][lane + 32] = o[h][0].y;
                        if (win > 64) {
                            T[h][lane + 64] = o[h][1].x;
                            T[h][lane + 96] = o[h][1].y;
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const float *t = T[h] + qi[h][m];
                        float a = grp[c0 + h][m];
                        a = fmaf(wv[h][m][0], t[0], a);
                        a = fmaf(wv[h][m][1], t[1], a);
                        if (!two[h]) {
#pragma unroll
                            for (int i = 2; i < NW; ++i)
                                a = fmaf(wv[h][m][i], lds_if(t + i, wv[h][m][i]), a);
                        }
                        grp[c0 + h][m] = a;
                    }
            }
            if (++ngrp == BP_GROUP || ib + sv + 1 == va1) flush(ib + sv + 1);
        }
        __syncwarp();  // the table and the row buffers are reused
    }
    if (S > 1) cl.sync();
    else __syncthreads();
    for (int col = warp * S + rank; col < BT * BT; col += 8 * S) {
        const int ix = x0 + (col & 7), jy = y0 + (col >> 3);
        if (ix >= g.nx || jy >= g.ny) continue;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int iz = 32 * m + lane;
            if (iz >= zn) continue;
            float2 *k = kh + col * SZ + iz;
            Kahan a;
            if (S == 1) {
                a.s = k->x;
            } else {
                for (int r = 0; r < S; ++r) {
                    const float2 t = *cl.map_shared_rank(k, r);
                    a.merge(t);
                }
            }
            float *o = vol + ((size_t)ix * g.ny + jy) * g.nz + z0 + iz;
            *o = accumulate ? *o + a.s : a.s;
        }
    }
    if (S > 1) cl.sync();  // no block leaves while its sums are read
}

template <int VEC, int M>
int launch_bp(const vg_dd3d_geom *g, const float *qw, const double *trig, int a0, int cnt, float *vol,
              cudaStream_t st) {
    constexpr size_t smem = (size_t)BT * BT * 32 * M * sizeof(float2) + 8 * sizeof(SfBpWarp);
    const long long tiles = (long long)ceil_div(g->nz, 32 * M) * ceil_div(g->ny, BT) * ceil_div(g->nx, BT);
    int S = 1;
    while (S < 8 && tiles * S < 3 * NSM && cnt >= 32 * S) S *= 2;
    int s = cuda_status(cudaFuncSetAttribute(sf3d_bp_kernel<VEC, M>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "sf3d_bp");
    if (s) return s;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(ceil_div(g->nz, 32 * M) * S, ceil_div(g->ny, BT), ceil_div(g->nx, BT));
    c.blockDim = dim3(256);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&c, sf3d_bp_kernel<VEC, M>, *g, qw, trig, a0, cnt, (int)(a0 > 0), vol),
                       "sf3d_bp");
}

// Columns over any number of u cells, slices over any number of v cells (a warp: 8
// columns of 32 slices, one view and column after the other).  The v cells that a
// column's slices reach pass through the warp's buffer in pieces, the column's u cells
// added up on the way; every lane then adds its slice's cells.  Up to 4 weights of a
// column and its v map come from a table as in the column kernel; of wider ones the lanes
// work out 32 weights at once.  Spare entries every 32 keep lanes 4, 8, 16 cells apart on
// different banks.  Cells of no weight or overlap are left out.  Sums: 16 views, then
// compensated.  128^3, 180 views, slices over 4 to 6 v cells: 8.1 -> 3.5 ms against the
// column kernel's per-voxel path, columns over 7 to 12 u cells 27 -> 10.4 (4 blocks per SM,
// with spills, 3.3 and 11.1).
constexpr int WIDE_ROWS = 480;
__device__ __forceinline__ int spare(int i) { return i + ((i >> 5) << 2); }
struct SfWideWarp {
    float T[WIDE_ROWS + WIDE_ROWS / 8];
    float4 w[4][BT];    // F1 l_phi0 / dv of u cells j0 .. j0 + 3
    float4 rec[4][BT];  // v cells per slice, Win's y and middle, j0 | count << 21
    float grp[BT][32];
    float2 kh[BT][32];  // (sum, compensation)
};

template <int VEC>
__global__ void __launch_bounds__(256, SF_WIDE_MINB)
sf3d_bp_wide_kernel(vg_dd3d_geom g, const float *__restrict__ qw, const double *__restrict__ trig, int a0, int cnt,
                    int accumulate, float *__restrict__ vol) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SfWideWarp &W = reinterpret_cast<SfWideWarp *>(smem4)[warp];
    const int z0 = blockIdx.x * 32, iy = blockIdx.y * BT + warp, x0 = blockIdx.z * BT;
    if (iy >= g.ny) return;  // no block barriers below
    const int zn = min(32, g.nz - z0), nc = min(BT, g.nx - x0);
    const float inv_du = 1.0f / g.du, U0 = uedge(g, 0);
    const float zd = (float)(z0 + (zn >> 1)) - 0.5f * g.nz;  // the middle slice's edge
    const float cv = 0.5f * g.nv - g.sv, ci = floorf(cv), cf = cv - ci;
    for (int c = 0; c < BT; ++c) {
        W.grp[c][lane] = 0.f;
        W.kh[c][lane] = make_float2(0.f, 0.f);
    }
    for (int ib = 0; ib < cnt; ib += 4) {
        {
            const int sv = lane >> 3, c = lane & 7;
            const float2 cs = view_cs(trig, a0 + min(ib + sv, cnt - 1));
            float w[BKU] = {0.f, 0.f, 0.f, 0.f};
            float B = 1.f;
            Win wn = {};
            int j0 = 0, n = 0;
            if (c < nc) {
                const SfCol C = sf_col(g, cs.x, cs.y, vox(g.d_pix, x0 + c, g.nx), vox(g.d_pix, iy, g.ny));
                const int ja = max((int)floorf((C.t0 - U0) * inv_du), 0);
                n = max(min((int)floorf((C.t3 - U0) * inv_du), g.nu - 1) - ja + 1, 0);
                j0 = min(ja, g.nu - 1);
                float e = trap_cum(uedge(g, j0), C);
                const float f = inv_du * C.lphi;
#pragma unroll
                for (int t = 0; t < BKU; ++t) {
                    const float h = trap_cum(uedge(g, j0 + t + 1), C);
                    w[t] = t < n ? (h - e) * f : 0.f;
                    e = h;
                }
                B = C.mz / g.dv;
                wn = win_at<1>(B, B * zd, cf, ci, zn);
            }
            W.w[sv][c] = make_float4(w[0], w[1], w[2], w[3]);
            W.rec[sv][c] = make_float4(B, wn.y, __int_as_float(max(min(wn.start + wn.mid, 1 << 29), -(1 << 29))),
                                       __int_as_float(j0 | min(n, BKU + 1) << 21));  // nu < 2^21
            __syncwarp();
        }
        const int nb = min(4, cnt - ib);
        for (int sv = 0; sv < nb; ++sv) {
            const float *q = qw + (size_t)(ib + sv) * g.nu * g.nv;
            for (int c = 0; c < nc; ++c) {
                const float4 rc = W.rec[sv][c];
                const int bits = __float_as_int(rc.w), mid = __float_as_int(rc.z);
                if (bits >> 21 == 0) continue;
                const float B = rc.x;
                const auto at = [&](int z) {  // slice z's first edge, in v cells from mid on
                    return fminf(fmaxf(fmaf(B, (float)(z - (zn >> 1)), rc.y), -1073741824.f), 1073741824.f);
                };
                const int z = min(lane, zn - 1);
                const float tl = at(z), th = at(z + 1), fl = floorf(tl), fh = floorf(th);
                const int r0 = mid + (int)fl, r1 = mid + (int)fh;
                const int la = max(__shfl_sync(0xffffffffu, r0, 0), 0) & ~(VEC - 1);
                const int le = min(__shfl_sync(0xffffffffu, r1, zn - 1) + 1, g.nv);
                const float w0 = fminf(B, (fl + 1.0f) - tl), w1 = fh > fl ? th - fh : 0.f;
                float s = 0.f;
                // the slices' sums of cells [l0, l0 + n) at T
                auto add = [&](int l0, int n) {
                    __syncwarp();
                    const int e = min(r1 - l0, n);
                    for (int i = max(r0 + 1 - l0, 0); i < e; ++i) s += W.T[spare(i)];
                    if ((unsigned)(r0 - l0) < (unsigned)n) s = fmaf(w0, W.T[spare(r0 - l0)], s);
                    if (w1 > 0.f && (unsigned)(r1 - l0) < (unsigned)n) s = fmaf(w1, W.T[spare(r1 - l0)], s);
                    __syncwarp();
                };
                if (bits >> 21 <= BKU) {
                    const float4 w = W.w[sv][c];
                    const float *qj = q + (size_t)(bits & 0x1fffff) * g.nv;
                    for (int l0 = la; l0 < le; l0 += WIDE_ROWS) {
                        const int n = min(WIDE_ROWS, le - l0);
                        for (int i = VEC * lane; i < n; i += 32 * VEC) {
                            const float *p = qj + l0 + i;
                            if (VEC == 4) {
                                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                                auto mac = [&](float x, const float *p) {
                                    const float4 f = __ldg(reinterpret_cast<const float4 *>(p));
                                    o = make_float4(fmaf(x, f.x, o.x), fmaf(x, f.y, o.y), fmaf(x, f.z, o.z),
                                                    fmaf(x, f.w, o.w));
                                };
                                if (w.x != 0.f) mac(w.x, p);
                                if (w.y != 0.f) mac(w.y, p + g.nv);
                                if (w.z != 0.f) mac(w.z, p + 2 * (size_t)g.nv);
                                if (w.w != 0.f) mac(w.w, p + 3 * (size_t)g.nv);
                                *reinterpret_cast<float4 *>(W.T + spare(i)) = o;
                            } else {
                                float o = w.x != 0.f ? w.x * __ldg(p) : 0.f;
                                if (w.y != 0.f) o = fmaf(w.y, __ldg(p + g.nv), o);
                                if (w.z != 0.f) o = fmaf(w.z, __ldg(p + 2 * (size_t)g.nv), o);
                                if (w.w != 0.f) o = fmaf(w.w, __ldg(p + 3 * (size_t)g.nv), o);
                                W.T[spare(i)] = o;
                            }
                        }
                        add(l0, n);
                    }
                } else {
                    const float2 cs = view_cs(trig, a0 + ib + sv);
                    const SfCol C = sf_col(g, cs.x, cs.y, vox(g.d_pix, x0 + c, g.nx), vox(g.d_pix, iy, g.ny));
                    const int jb = min((int)floorf((C.t3 - U0) * inv_du), g.nu - 1);
                    for (int j0 = bits & 0x1fffff; j0 <= jb; j0 += 32) {
                        const int nj = min(32, jb - j0 + 1);
                        const float w =
                            lane < nj ? uweight(C, uedge(g, j0 + lane), uedge(g, j0 + lane + 1), inv_du) : 0.f;
                        for (int l0 = la; l0 < le; l0 += WIDE_ROWS) {
                            const int n = min(WIDE_ROWS, le - l0);
                            for (int i = 0; i < n; i += 32) {
                                const float *p = q + (size_t)j0 * g.nv + (l0 + min(i + lane, n - 1));
                                float o = 0.f;
#pragma unroll 4
                                for (int t = 0; t < nj; ++t, p += g.nv) {
                                    const float wt = __shfl_sync(0xffffffffu, w, t);
                                    if (wt != 0.f) o = fmaf(wt, __ldg(p), o);
                                }
                                W.T[spare(i + lane)] = o;
                            }
                            add(l0, n);
                        }
                    }
                }
                W.grp[c][lane] += s;
            }
        }
        if ((ib & 15) == 12 || ib + 4 >= cnt)
            for (int c = 0; c < nc; ++c) {
                Kahan k;
                k.s = W.kh[c][lane].x; k.c = W.kh[c][lane].y;
                k.add(W.grp[c][lane]);
                W.kh[c][lane] = make_float2(k.s, k.c);
                W.grp[c][lane] = 0.f;
            }
        __syncwarp();  // the table is reused
    }
    if (lane < zn)
        for (int c = 0; c < nc; ++c) {
            float *o = vol + ((size_t)(x0 + c) * g.ny + iy) * g.nz + z0 + lane;
            *o = accumulate ? *o + W.kh[c][lane].x : W.kh[c][lane].x;
        }
}

template <int VEC>
int launch_bp_wide(const vg_dd3d_geom *g, const float *qw, const double *trig, int a0, int cnt, float *vol,
                   cudaStream_t st) {
    constexpr size_t smem = 8 * sizeof(SfWideWarp);
    int s = cuda_status(cudaFuncSetAttribute(sf3d_bp_wide_kernel<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem), "sf3d_bp_wide");
    if (s) return s;
    dim3 grid(ceil_div(g->nz, 32), ceil_div(g->ny, BT), ceil_div(g->nx, BT));
    sf3d_bp_wide_kernel<VEC><<<grid, 256, smem, st>>>(*g, qw, trig, a0, cnt, (int)(a0 > 0), vol);
    return launch_status("sf3d_bp_wide");
}

int check(const vg_dd3d_geom *g) {
    VG_REQUIRE(g, "sf3d: null geometry");
    VG_REQUIRE(g->nx > 0 && g->ny > 0 && g->nz > 0 && g->na > 0 && g->nu > 0 && g->nv > 0,
               "sf3d: sizes must be positive");
    VG_REQUIRE(g->na < 65536 && ceil_div(g->nx, BT) < 65536 && ceil_div(g->ny, BT) < 65536 &&
                   ceil_div(g->nu, 32) < 65536, "sf3d: sizes too large");
    VG_REQUIRE(g->nx <= 2048 && g->ny <= 2048, "sf3d: nx and ny at most 2048");
    VG_REQUIRE((double)g->nx * g->ny * (g->nz + 1) < 2147483648.0, "sf3d: volume above 2^31 voxels");
    VG_REQUIRE(g->du > 0.f && g->dv > 0.f && g->d_pix > 0.f && g->DSO > 0.f && g->DSD > 0.f,
               "sf3d: pitches and distances must be positive");
    // every voxel in front of the source (its footprint's projections are
    // then finite): the volume's half diagonal in the plane below DSO
    const float hx = 0.5f * g->nx * g->d_pix, hy = 0.5f * g->ny * g->d_pix;
    VG_REQUIRE(hx * hx + hy * hy < g->DSO * g->DSO,
               "sf3d: the volume must lie inside the source circle (half diagonal below DSO)");
    return VG_OK;
}

constexpr size_t SF_CHUNK_BYTES = (size_t)256 << 20;

size_t chunk_views(const vg_dd3d_geom *g) {
    const size_t per = (size_t)g->nu * g->nv * sizeof(float);
    size_t n = SF_CHUNK_BYTES / per;
    if (n < 1) n = 1;
    if (n > (size_t)g->na) n = g->na;
    return n;
}

size_t bp_ws_bytes(const vg_dd3d_geom *g) {
    return chunk_views(g) * (size_t)g->nu * g->nv * sizeof(float);
}

// the forward projection's running sums over z (LONG); asked for in every geometry, as
// callers size and check their workspace by it
size_t fp_ws_bytes(const vg_dd3d_geom *g) {
    return (size_t)g->nx * g->ny * (g->nz + 1) * sizeof(float);
}

}  // namespace

extern "C" size_t vg_sf3d_workspace_bytes(const vg_dd3d_geom *g) {
    if (check(g)) return 0;
    const size_t f = fp_ws_bytes(g), b = bp_ws_bytes(g);
    return f > b ? f : b;
}

extern "C" int vg_sf3d_fp(const vg_dd3d_geom *g, const float *vol, const double *trig, float *sino,
                          void *workspace, size_t workspace_bytes, void *stream) {
    int st = check(g);
    if (st) return st;
    VG_REQUIRE(vol && trig && sino, "sf3d_fp: null pointer");
    const size_t need = fp_ws_bytes(g);
    VG_REQUIRE(workspace && workspace_bytes >= need,
               "sf3d_fp: workspace of %zu bytes needed (vg_sf3d_workspace_bytes)", need);
    VG_REQUIRE(((uintptr_t)workspace & 3) == 0, "sf3d_fp: workspace must be 4-byte aligned");
    cudaStream_t s = as_stream(stream);
    // 96 or 64 v cells per warp while the slices under them fit a row buffer, by the
    // smallest magnification in the volume; 96 unless the detector's last tile is
    // emptier for it; 16-byte loads where columns are aligned
    const double r = 0.5 * hypot((double)g->nx, (double)g->ny) * g->d_pix;
    const double bmax = (g->DSO + r) / g->DSD * g->dv / g->d_pix;
    const bool vec = g->nz % 4 == 0 && ((uintptr_t)vol & 15) == 0;
    if (g->nv > 32 && 96.0 * bmax + 9.0 <= BW && 96 * ceil_div(g->nv, 96) <= 1.15 * 64 * ceil_div(g->nv, 64))
        return vec ? launch_fp<4, 3>(g, vol, trig, sino, s) : launch_fp<1, 3>(g, vol, trig, sino, s);
    if (g->nv > 32 && 64.0 * bmax + 9.0 <= BW)
        return vec ? launch_fp<4, 2>(g, vol, trig, sino, s) : launch_fp<1, 2>(g, vol, trig, sino, s);
    if (32.0 * bmax + 9.0 <= BW)
        return vec ? launch_fp<4, 1>(g, vol, trig, sino, s) : launch_fp<1, 1>(g, vol, trig, sino, s);
    // v cells over more slices: running sums of about a cell's slices, so that a cell
    // meets one end of them and carries their rounding
    int lz = 2;
    while (lz < 5 && (1 << lz) < bmax) ++lz;
    float *zs = static_cast<float *>(workspace);
    sf3d_zsums<<<1216, 256, 0, s>>>(*g, vol, lz, zs);
    st = launch_status("sf3d_zsums");
    if (st) return st;
    return g->nv > 32 ? launch_fp<1, 2, true>(g, vol, trig, sino, s, zs, lz)
                      : launch_fp<1, 1, true>(g, vol, trig, sino, s, zs, lz);
}

extern "C" int vg_sf3d_bp(const vg_dd3d_geom *g, const float *sino, const double *trig, float *vol,
                          void *workspace, size_t workspace_bytes, void *stream) {
    int st = check(g);
    if (st) return st;
    VG_REQUIRE(sino && trig && vol, "sf3d_bp: null pointer");
    const size_t nch = chunk_views(g);
    const size_t need = bp_ws_bytes(g);
    VG_REQUIRE(workspace && workspace_bytes >= need,
               "sf3d_bp: workspace of %zu bytes needed (vg_sf3d_workspace_bytes)", need);
    cudaStream_t s = as_stream(stream);
    float *qw = static_cast<float *>(workspace);
    // 64 slices per warp while the cells they project to fit a row buffer, by the
    // largest magnification in the volume; 16-byte loads where rows are aligned
    const double r = 0.5 * hypot((double)g->nx, (double)g->ny) * g->d_pix;
    const double bmax = g->DSD / (g->DSO - fmin(r, 0.999 * g->DSO)) * g->d_pix / g->dv;
    const bool m2 = g->nz > 32 && 64.0 * bmax + 9.0 <= BW;
    const bool vec = g->nv % 4 == 0 && ((uintptr_t)qw & 15) == 0;
    // the wide kernel where cells do not fit a row buffer, or columns reach 4.2 u cells, by
    // the widest at the near side (128^3, 120 views: 1.7 against 1.9 ms at 4.0, 3.3 against
    // 2.5 at 4.2)
    const bool wide = (!m2 && 32.0 * bmax + 9.0 > BW) || 1.415 * bmax * g->dv / g->du > 4.2;
    auto bp = wide ? (vec ? launch_bp_wide<4> : launch_bp_wide<1>)
              : m2 ? (vec ? launch_bp<4, 2> : launch_bp<1, 2>) : (vec ? launch_bp<4, 1> : launch_bp<1, 1>);
    for (int a0 = 0; a0 < g->na; a0 += (int)nch) {
        const int cnt = (int)((size_t)(g->na - a0) < nch ? (size_t)(g->na - a0) : nch);
        sf3d_weight<<<1216, 256, 0, s>>>(*g, sino, a0, cnt, qw);
        st = launch_status("sf3d_weight");
        if (st) return st;
        st = bp(g, qw, trig, a0, cnt, vol, s);
        if (st) return st;
    }
    return VG_OK;
}
