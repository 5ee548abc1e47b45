// 3D cone-beam distance-driven projector pair, gather form.
//
// vir's cone sweep (sys_mat/dd.py:285-468, geometry 589-645, wrappers
// 815-888) weights voxel (k along the driving axis, line io, slice iz) into
// bin (iu, iv) by
//     scale(io) * |[P_k, P_k+1] ∩ [U_iu, U_iu+1]| * |zmag(io) [z_iz, z_iz+1] ∩ [V_iv, V_iv+1]|
// with P the fan projection of the driving edges on line io (as in 2D),
// zmag(io) = DSD / (DSO - o_centre(io)) and z_iz = d_pix (iz - nz/2); FP
// returns sino * d_pix^2 / (du dv), BP returns img / (na d_pix).  The u and v
// factors are separable per line, so each (bin, line) or (voxel, view) pair
// touches only the 1-3 pixels x 1-2 slices (or bins) its intervals overlap.
// (vir's FP reuses a stale u buffer across lines, dd.py:300,335; this is the
// overlap integral that sweep intends.)
//
//  dd3d_prep: per (view, line) the scale and z magnification (workspace).
//  FP: warp = 8 u cells of one view, lanes along v; walks the lines; the
//      pixels under a cell come from the exact inverse of the edge projection.
//  BP: warp = 8 columns of a pixel line, lanes along z; walks the views.
#include <cooperative_groups.h>
#include <math.h>

#include "vg_common.cuh"

namespace {

using namespace vg;
namespace cg = cooperative_groups;

struct View3 {
    float pd, od, po, oo, tabs;
    int xdrv;
};

__device__ __forceinline__ View3 view3(const double *trig, int ia) {
    View3 v;
    const float c = (float)__ldg(trig + 2 * ia), s = (float)__ldg(trig + 2 * ia + 1);
    v.xdrv = fabsf(s) >= fabsf(c);
    if (v.xdrv) { v.pd = -s; v.od = c; v.po = c; v.oo = s; v.tabs = fabsf(s); }
    else        { v.pd = c;  v.od = s; v.po = -s; v.oo = c; v.tabs = fabsf(c); }
    return v;
}

__device__ __forceinline__ float cen(float d, int i, int n) { return d * ((float)i + 0.5f - 0.5f * n); }
__device__ __forceinline__ float edg(float d, int i, int n) { return d * ((float)i - 0.5f * n); }

// Pole of the inverse edge map (u of rays parallel to the lines): whether it
// lies in [a, b].  It is outside every line's shadow, but a detector that
// reaches DSD from the centre can contain it; ranges found through the
// inverse map are then not trusted on an interval holding it.
__device__ __forceinline__ bool pole_in(const vg_dd3d_geom &g, const View3 &v, float a, float b) {
    if (v.od == 0.f) return false;
    const float Up = -g.DSD * v.pd / v.od;
    return Up >= fminf(a, b) && Up <= fmaxf(a, b);
}

__device__ __forceinline__ float projU(const vg_dd3d_geom &g, const View3 &v, float cp, float co,
                                       float b) {
    return __fdividef(g.DSD * fmaf(v.pd, b, cp), g.DSO - fmaf(v.od, b, co));
}

// Workspace: tab[na][max(nx, ny)] float2 (scale, zmag) per (view, line),
// then, 16-byte aligned, vf[na][2] float4 per view: (pd, od, po, oo) and
// (|trig|, xdrv, 0, 0), the float view geometry of view3, then
// bt[na][max(nx, ny)] double2, the v cells per slice and the slices per v cell
// of every line.
size_t tab_bytes(const vg_dd3d_geom *g) {
    const int nm = g->nx > g->ny ? g->nx : g->ny;
    return ((size_t)g->na * nm * 2 * sizeof(float) + 15) & ~(size_t)15;
}

size_t vf_bytes(const vg_dd3d_geom *g) { return (size_t)g->na * 2 * sizeof(float4); }

size_t ws_bytes(const vg_dd3d_geom *g) {
    const int nm = g->nx > g->ny ? g->nx : g->ny;
    return tab_bytes(g) + vf_bytes(g) + (size_t)g->na * nm * sizeof(double2);
}

struct Ws3 {
    const float2 *tab;
    const float4 *vf;
    const double2 *bt;
};

Ws3 ws_of(const vg_dd3d_geom *g, const void *ws) {
    const char *p = static_cast<const char *>(ws);
    return {reinterpret_cast<const float2 *>(p), reinterpret_cast<const float4 *>(p + tab_bytes(g)),
            reinterpret_cast<const double2 *>(p + tab_bytes(g) + vf_bytes(g))};
}

__device__ __forceinline__ View3 view_f(const float4 *__restrict__ vf, int ia) {
    const float4 a = vf[2 * ia], b = vf[2 * ia + 1];
    View3 v;
    v.pd = a.x; v.od = a.y; v.po = a.z; v.oo = a.w; v.tabs = b.x; v.xdrv = b.y != 0.f;
    return v;
}

// tab[ia][io] = (scale, zmag); vf[ia] = float view geometry; bt[ia][io] =
// zmag d_pix / dv and its reciprocal in FP64, from which a tile's first row is
// found without the rounding of a float32 coordinate
__global__ void dd3d_prep(vg_dd3d_geom g, const double *__restrict__ trig, float2 *__restrict__ tab,
                          float4 *__restrict__ vf, double2 *__restrict__ bt) {
    const int ia = blockIdx.x;
    const View3 v = view3(trig, ia);
    const int no = v.xdrv ? g.ny : g.nx;
    const int nm = g.nx > g.ny ? g.nx : g.ny;
    if (threadIdx.x == 0) {
        vf[2 * ia] = make_float4(v.pd, v.od, v.po, v.oo);
        vf[2 * ia + 1] = make_float4(v.tabs, v.xdrv ? 1.f : 0.f, 0.f, 0.f);
    }
    for (int io = threadIdx.x; io < no; io += blockDim.x) {
        const float c = cen(g.d_pix, io, no);
        const float cp = v.po * c, co = v.oo * c;
        const float a = g.DSO - co;
        tab[(size_t)ia * nm + io] = make_float2(sqrtf(a * a + cp * cp) / (a * v.tabs), g.DSD / a);
        const double cd = (double)g.d_pix * ((double)io + 0.5 - 0.5 * no);
        const double b = (double)g.DSD * g.d_pix / ((double)g.dv * (g.DSO - v.oo * cd));
        bt[(size_t)ia * nm + io] = make_double2(b, 1.0 / b);
    }
}

__device__ __forceinline__ float ufloor_edge(const vg_dd3d_geom &g, int j) {
    return g.du * ((float)j - 0.5f * g.nu + g.su);
}
__device__ __forceinline__ float vfloor_edge(const vg_dd3d_geom &g, int j) {
    return g.dv * ((float)j - 0.5f * g.nv + g.sv);
}

// One cell's share of one line, straight from global memory (any geometry).
__device__ __noinline__ float fp_cell_line(const vg_dd3d_geom &g, const View3 &v, const float *__restrict__ vol,
                              size_t sk, size_t so, int nd, int io, float cp, float co, float zmag,
                              float Ul, float Ur, float Vl, float Vr) {
    const float inv_d = 1.0f / g.d_pix;
    const float rl = 1.0f / (g.DSD * v.pd + Ul * v.od), rr = 1.0f / (g.DSD * v.pd + Ur * v.od);
    const float kl = fmaf(Ul, g.DSO - co, -g.DSD * cp) * rl * inv_d + 0.5f * nd;
    const float kr = fmaf(Ur, g.DSO - co, -g.DSD * cp) * rr * inv_d + 0.5f * nd;
    const bool pole = pole_in(g, v, Ul, Ur);
    const int k0 = pole ? 0 : max(0, (int)floorf(fminf(kl, kr)));
    const int k1 = pole ? nd - 1 : min(nd - 1, (int)floorf(fmaxf(kl, kr)));
    const float izl = Vl / (zmag * g.d_pix) + 0.5f * g.nz;
    const float izr = Vr / (zmag * g.d_pix) + 0.5f * g.nz;
    const int z0 = max(0, (int)floorf(izl)), z1 = min(g.nz - 1, (int)floorf(izr));
    float part = 0.f;
    if (k0 > k1 || z0 > z1) return part;
    float pa = projU(g, v, cp, co, edg(g.d_pix, k0, nd));
    for (int k = k0; k <= k1; ++k) {
        const float pb = projU(g, v, cp, co, edg(g.d_pix, k + 1, nd));
        const float ou = fminf(fmaxf(pa, pb), Ur) - fmaxf(fminf(pa, pb), Ul);
        pa = pb;
        if (ou <= 0.f) continue;
        const float *col = vol + k * sk + io * so;
        float colsum = 0.f;
        for (int iz = z0; iz <= z1; ++iz) {
            const float zl = zmag * edg(g.d_pix, iz, g.nz), zr = zmag * edg(g.d_pix, iz + 1, g.nz);
            const float ov = fminf(zr, Vr) - fmaxf(zl, Vl);
            if (ov > 0.f) colsum = fmaf(__ldg(col + iz), ov, colsum);
        }
        part = fmaf(colsum, ou, part);
    }
    return part;
}

// --- both kernels: overlaps applied one axis after the other ---------------
//
// A warp owns 8 output columns (BP: pixel columns of one line; FP: u cells of
// one view) and 32 M outputs along each (slices; v cells).  For one line and
// view every output is a sum over 1-4 input columns (detector columns; pixel
// columns) times a u-overlap, and over 1-5 input rows (v cells; slices) times
// a v-overlap, and the v-overlaps are the same for all 8 columns.  So instead
// of a 3 x 3 gather per output:
//   u: over the window of rows that its outputs reach, the warp adds the input
//      columns -- one aligned 16-byte load per 4 rows -- into a row buffer in
//      shared memory; output columns are taken in pairs, which mostly share an
//      input column;
//   v: every output adds its rows of that buffer, with v-overlaps that stay in
//      registers for the line.
// Rows are counted in input cells from the one at the middle of the tile's
// outputs, which is found in FP64, so a cell edge is an integer and an output's
// edge carries the rounding of its distance from there, however short the tile.
// The u-overlaps of 4 lines or views are
// tabulated at once (lane = line or view x column) in the warp's own shared
// memory: the warps of a block do not wait for each other.
//
// What bounds it: instruction issue (FP 56 %, BP 60 %) and the L1 data pipe (54 and
// 79 %, from the v step, whose lanes are 1.15 rows apart and so hit a bank twice)
// together.  Against the 3 x 3 gather through tables of all cells' overlaps, at
// 256^3 voxels, 360 views of 512 x 384: FP 22.4 -> 13.1 ms, BP 17.3 -> 9.3 ms;
// 512^3, 720 views of 1024 x 768: 634 -> 418 ms the pair.  Measured at 256^3 and
// not kept: the detector window of a BP tile copied into shared memory by the
// block, with 16-byte reads per column 15.6 ms, with 4 columns' rows side by
// side 11.0 ms; that layout on global loads 12.6 ms.
constexpr int BT = 8;    // columns per warp
constexpr int BW = 128;  // rows of one column buffer
constexpr int FP_GROUP = 16, BP_GROUP = 16;  // lines, views summed in registers before the running sum

// a pair's columns start one input column apart and have 2-3 each
constexpr int SHARED = 1 << 31;

struct WarpBuf {
    float T[2][2][BW];
    // of 4 lines or views, columns in input order within a pair:
    float4 uw[4][BT];  // overlaps with 3 input columns, (bits) the first | count << 20
                       // | SHARED in a pair's first column
    float w3[4][BT];   // overlap with a fourth
    float4 line[4];    // of the v step, see Line
};

// The rows of zn outputs, b input rows each, the middle one (zn / 2) starting at row
// t of the input (n rows): they are counted from row c = floor(t), and the window
// that is staged starts at a multiple of 4 at or below the first output's row, found
// with the expression of Strip::init.  Packed as (b, t - c, window's start + falling
// input order, c - start | rows of the window << 12), or, where the rows do not fit a
// column buffer or one output's NW, (b, t - c, falling input order, c) for long_pair.
struct Line {
    float b, y;
    int start, mid, rows;

    template <int NW>
    __device__ __forceinline__ bool fits() const { return b <= NW - 1.0f && rows <= BW - NW + 1; }
    __device__ __forceinline__ float4 pack(int rev, bool fit) const {
        return make_float4(b, y, __int_as_float(fit ? start + rev : rev),
                           __int_as_float(fit ? mid | rows << 12 : start + mid));
    }
};
__device__ __forceinline__ Line line_at(double b, double t, int zn) {
    Line l;
    const int c = __double2int_rd(t);
    const float lo = -(float)(zn >> 1);
    l.b = (float)b;
    l.y = fminf((float)(t - c), 0.99999994f);  // below 1, so that the start is at c at most
    l.start = (c + __float2int_rd(fmaf(l.b, lo, l.y))) & ~3;
    l.mid = c - l.start;
    l.rows = l.mid + __float2int_rd(fmaf(l.b, (float)zn + lo, l.y)) + 1;
    return l;
}

// One line and view of a warp.  VEC: floats per input load (4 needs input
// columns that start on 16-byte boundaries).  M = 2 takes outputs of up to 2
// rows, M = 1 of up to 4.
template <int VEC, int M>
struct Strip {
    static constexpr int NW = M >= 2 ? 3 : 5, NV = 4 / VEC;
    float w[M][NW];    // v-overlaps of this lane's outputs (rows)
    int qa[M], qb[M];  // their first row in the buffers of a pair's columns
    int vo[NV];        // rows this lane loads
    const char *in;    // the input, from this lane's first row on (VEC 4)
    unsigned st;       // bytes between input columns
    int win;
    bool two;

    // packed Line ln, zn outputs, an input of n rows
    __device__ __forceinline__ void init(const float *src, unsigned stride, int lane, float4 ln, int zn, int n) {
        const int vs = __float_as_int(ln.z) & ~3, sw = __float_as_int(ln.z) & 1;
        const int mid = __float_as_int(ln.w) & 0xfff;
        float over = 0.f;
        int qf[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float zm = (float)(32 * m + lane - (zn >> 1));
            const float tl = fmaf(ln.x, zm, ln.y), th = fmaf(ln.x, zm + 1.0f, ln.y);
            const float tf = floorf(tl);
            w[m][0] = fminf(ln.x, (tf + 1.0f) - tl);  // all of an output inside one row: its size, unrounded
#pragma unroll
            for (int t = 1; t < NW; ++t) w[m][t] = __saturatef(th - (tf + (float)t));
            if (32 * m + lane < zn) over = fmaxf(over, th - tf);
            qf[m] = (int)tf + mid;
            const int q = min(qf[m], BW - NW);  // outputs past the end read anything
            qa[m] = q + (sw ? BW : 0);
            qb[m] = q + (sw ? 0 : BW);
        }
        two = !__any_sync(0xffffffffu, over > 2.0f);
        // rows are clamped to the window and the input; rows outside it weigh nothing
        win = (__float_as_int(ln.w) >> 12) + NW - 1;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int v = vs + min(VEC == 4 ? 4 * lane : lane + 32 * i, (win - 1) & ~(VEC - 1));
            vo[i] = min(max(v, 0), n - VEC);
        }
        in = reinterpret_cast<const char *>(VEC == 4 ? src + vo[0] : src);
        st = 4 * stride;
        if (vs < 0 || vs + win > n) {
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int t = 0; t < NW; ++t)
                    if ((unsigned)(qf[m] + vs + t) >= (unsigned)n) w[m][t] = 0.f;
        }
    }

    __device__ __forceinline__ void load(unsigned j, float2 (&r)[2]) const {  // of input column j
        const char *q = ptr_at(in, j, st);
        if (VEC == 4) {
            const float4 f = __ldg(reinterpret_cast<const float4 *>(q));
            r[0] = make_float2(f.x, f.y);
            r[1] = make_float2(f.z, f.w);
        } else {
            const float *f = reinterpret_cast<const float *>(q);
            r[0] = make_float2(__ldg(f + vo[0]), __ldg(f + vo[1 & (NV - 1)]));
            if (win > 64) r[1] = make_float2(__ldg(f + vo[2 & (NV - 1)]), __ldg(f + vo[3 & (NV - 1)]));
        }
    }
    static __device__ __forceinline__ void mul(float x, const float2 (&r)[2], float2 (&o)[2]) {
        o[0] = pk_mul(make_float2(x, x), r[0]);
        o[1] = pk_mul(make_float2(x, x), r[1]);
    }
    static __device__ __forceinline__ void mac(float x, const float2 (&r)[2], float2 (&o)[2]) {
        o[0] = pk_fma(make_float2(x, x), r[0], o[0]);
        o[1] = pk_fma(make_float2(x, x), r[1], o[1]);
    }
    __device__ __forceinline__ void put(int lane, float *t, const float2 (&o)[2]) const {
        if (VEC == 4) {
            if (4 * lane < win)
                *reinterpret_cast<float4 *>(t + 4 * lane) = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
        } else {
            t[lane] = o[0].x;
            t[lane + 32] = o[0].y;
            if (win > 64) {
                t[lane + 64] = o[1].x;
                t[lane + 96] = o[1].y;
            }
        }
    }
    // this lane's outputs of one column: its rows at T + q
    __device__ __forceinline__ void rows(const float *T, const int (&q)[M], float (&grp)[M]) const {
#pragma unroll
        for (int m = 0; m + 1 < M; m += 2) {
            const float *t0 = T + q[m], *t1 = T + q[m + 1];
            float2 a = make_float2(grp[m], grp[m + 1]);
            a = pk_fma(make_float2(w[m][0], w[m + 1][0]), make_float2(t0[0], t1[0]), a);
            a = pk_fma(make_float2(w[m][1], w[m + 1][1]), make_float2(t0[1], t1[1]), a);
            if (!two) {  // a third row is read only by the outputs that have one
                const float2 x = make_float2(lds_if(t0 + 2, w[m][2]), lds_if(t1 + 2, w[m + 1][2]));
                a = pk_fma(make_float2(w[m][2], w[m + 1][2]), x, a);
            }
            grp[m] = a.x;
            grp[m + 1] = a.y;
        }
        if (M & 1) {
            const float *t = T + q[M - 1];
            float a = grp[M - 1];
            a = fmaf(w[M - 1][0], t[0], a);
            a = fmaf(w[M - 1][1], t[1], a);
            if (!two) {
#pragma unroll
                for (int i = 2; i < NW; ++i) a = fmaf(w[M - 1][i], lds_if(t + i, w[M - 1][i]), a);
            }
            grp[M - 1] = a;
        }
    }

    // output columns c, c + 1 of table row sv
    __device__ __forceinline__ void pair(WarpBuf &W, int sv, int c, int lane, float (&ga)[M],
                                         float (&gb)[M]) const {
        float (*T)[BW] = W.T[(c >> 1) & 1];
        const float4 el = W.uw[sv][c], eh = W.uw[sv][c + 1];
        const int bl = __float_as_int(el.w), bh = __float_as_int(eh.w);
        const unsigned j = bl & 0xfffff;
        float2 ol[2], oh[2], r0[2], r1[2];
        if (bl < 0) {  // SHARED: 3 loads for 2 x 2
            float2 r2[2];
            load(j, r0);
            load(j + 1, r1);
            load(j + 2, r2);
            mul(el.x, r0, ol);
            mac(el.y, r1, ol);
            mul(eh.x, r1, oh);
            mac(eh.y, r2, oh);
            if (bl & 1 << 20) mac(el.z, r2, ol);
            if (bh & 1 << 20) {
                load(j + 3, r0);
                mac(eh.z, r0, oh);
            }
        } else {
            const int nl = bl >> 20, nh = bh >> 20;
            const unsigned k = bh & 0xfffff;
            float2 r2[2], r3[2];
            load(j, r0);
            load(j + (nl > 1), r1);
            load(k, r2);
            load(k + (nh > 1), r3);
            mul(el.x, r0, ol);
            mac(el.y, r1, ol);
            mul(eh.x, r2, oh);
            mac(eh.y, r3, oh);
            if (nl > 2) {
                load(j + 2, r0);
                mac(el.z, r0, ol);
            }
            if (nh > 2) {
                load(k + 2, r2);
                mac(eh.z, r2, oh);
            }
            if (nl > 3) {
                load(j + 3, r1);
                mac(W.w3[sv][c], r1, ol);
            }
            if (nh > 3) {
                load(k + 3, r3);
                mac(W.w3[sv][c + 1], r3, oh);
            }
            // a column beside the input takes nothing from its nearest input column
            if (nl == 0) ol[0] = ol[1] = make_float2(0.f, 0.f);
            if (nh == 0) oh[0] = oh[1] = make_float2(0.f, 0.f);
        }
        put(lane, T[0], ol);
        put(lane, T[1], oh);
        __syncwarp();
        rows(T[0], qa, ga);
        rows(T[0], qb, gb);
    }
};

// Table entry of one output column (lane, slot = its place in input order
// within a pair): n <= 4 input columns from js on with overlaps w.
__device__ __forceinline__ void put_column(WarpBuf &W, int sv, int slot, const float (&w)[4], int js, int n,
                                           bool store = true) {
    const int js2 = __shfl_xor_sync(0xffffffffu, js, 1), n2 = __shfl_xor_sync(0xffffffffu, n, 1);
    const bool shared = !(slot & 1) && js2 == js + 1 && (n & ~1) == 2 && (n2 & ~1) == 2;
    if (!store) return;
    W.uw[sv][slot] = make_float4(w[0], w[1], w[2], __int_as_float(js | n << 20 | (shared ? SHARED : 0)));
    W.w3[sv][slot] = w[3];
}

// A pair's outputs on a line whose rows do not fit Strip: the rows in pieces of a
// column buffer, every output over its rows of each piece.
template <int M>
struct LongPair {
    float a[M], b[M];  // of output columns c and c + 1
};
template <int M>
__device__ __noinline__ LongPair<M> long_pair(WarpBuf &W, int sv, int c, const float *src, size_t stride, int zn,
                                              int n) {
    const int lane = threadIdx.x & 31;
    const float4 ln = W.line[sv];
    const int rev = __float_as_int(ln.z) & 1, mid = max(min(__float_as_int(ln.w), 1 << 29), -(1 << 29));
    const auto at = [&](int z) {  // output z's first edge, from row mid on
        return fminf(fmaxf(fmaf(ln.x, (float)(z - (zn >> 1)), ln.y), -1073741824.f), 1073741824.f);
    };
    const auto row = [&](int z) { return mid + __float2int_rd(at(z)); };
    LongPair<M> p;
#pragma unroll
    for (int m = 0; m < M; ++m) p.a[m] = p.b[m] = 0.f;
    const int r1 = min(row(zn) + 1, n);
    for (int r0 = max(row(0), 0); r0 < r1; r0 += BW) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 e = W.uw[sv][c + h];
            const int bits = __float_as_int(e.w), nc = bits >> 20 & 7;
            const float *q = src + (size_t)(bits & 0xfffff) * stride;
            const float w[4] = {e.x, e.y, e.z, W.w3[sv][c + h]};
            for (int i = lane; i < BW; i += 32) {
                float o = 0.f;
                if (r0 + i < r1)
                    for (int t = 0; t < nc; ++t) o = fmaf(w[t], __ldg(q + t * stride + (r0 + i)), o);
                W.T[0][h][i] = o;
            }
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int z = 32 * m + lane;
            if (z >= zn) continue;
            const float tl = at(z), th = at(z + 1);
            const int e = min(min(mid + __float2int_rd(th) + 1, r0 + BW), r1);
            for (int r = max(row(z), r0); r < e; ++r) {
                const float x = (float)(r - mid), ov = fminf(th, x + 1.0f) - fmaxf(tl, x);
                if (ov > 0.f) {
                    p.a[m] = fmaf(ov, W.T[0][rev][r - r0], p.a[m]);
                    p.b[m] = fmaf(ov, W.T[0][rev ^ 1][r - r0], p.b[m]);
                }
            }
        }
        __syncwarp();
    }
    return p;
}

// Forward projection.  Block = one view, 32 u cells x 32 M v cells; a warp
// owns 8 u cells and walks the lines of the volume, 4 at a time.  The pixel
// columns under a u cell come from the exact inverse of the edge projection.
// WIDE: lines where a u cell overlaps more than 4 pixels take 4 at a time, those
// where the tile's v cells overlap more slices than a column buffer holds long_pair;
// else such lines, few then, take the per-cell global path.  Sums: 16
// lines in registers, then a second running sum in shared memory.  At 128
// registers 4 blocks of 4 warps fit an SM: 13.1 ms at 256^3 (5 blocks, with
// spills, 13.8 ms; 3 15.0 ms); with 64 v cells per warp 16.0 ms.
constexpr int FPW = 4;       // warps per block
constexpr int FP_MINB = 4;
// MODE 0: projection; 1: SIRT residual epilogue
template <int MODE, int VEC, int M, bool WIDE>
__global__ void __launch_bounds__(32 * FPW, FP_MINB)
dd3d_fp_kernel(vg_dd3d_geom g, const float *__restrict__ vol, const float4 *__restrict__ vf,
               const float2 *__restrict__ tab, const double2 *__restrict__ bt, float *__restrict__ sino,
               const float *__restrict__ y, const float *__restrict__ inv_w) {
    constexpr int SZ = 32 * M;
    extern __shared__ float4 smem4[];
    const int ia = blockIdx.z, v0 = blockIdx.x * SZ;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = (blockIdx.y * FPW + warp) * BT;
    float *acc = reinterpret_cast<float *>(smem4) + warp * BT * SZ + lane;  // [BT][SZ] of this warp
    WarpBuf &W = reinterpret_cast<WarpBuf *>(reinterpret_cast<float *>(smem4) + FPW * BT * SZ)[warp];
    if (u0 >= g.nu) return;  // no block barriers below
    const View3 v = view_f(vf, ia);
    const int nd = v.xdrv ? g.nx : g.ny, no = v.xdrv ? g.ny : g.nx;
    const int nm = g.nx > g.ny ? g.nx : g.ny;
    const size_t sk = v.xdrv ? (size_t)g.ny * g.nz : (size_t)g.nz;  // stride of k
    const size_t so = v.xdrv ? (size_t)g.nz : (size_t)g.ny * g.nz;  // stride of io
    const float inv_d = 1.0f / g.d_pix;
    const int zn = min(SZ, g.nv - v0);
    const double vd = (double)(v0 + (zn >> 1)) - 0.5 * g.nv + (double)g.sv;  // the middle v cell's edge
    // this lane's u cell in the table (slot order: a pair's pixels ascending)
    const bool rev = v.pd < 0.f;
    const int ls = lane >> 3, cs = lane & 7, iu = u0 + (cs ^ (int)rev);
    const float Ul = ufloor_edge(g, iu), Ur = ufloor_edge(g, iu + 1);
    const float rl = 1.0f / (g.DSD * v.pd + Ul * v.od), rr = 1.0f / (g.DSD * v.pd + Ur * v.od);
    const bool cell = iu < g.nu, pole = cell && pole_in(g, v, Ul, Ur);
    const bool big = sk >= (1u << 30);  // byte strides are 32-bit below
    float grp[BT][M];
#pragma unroll
    for (int c = 0; c < BT; ++c)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            grp[c][m] = 0.f;
            acc[c * SZ + 32 * m] = 0.f;
        }
    // pixels under this lane's u cell on line io: their number, and from the k0-th on the
    // overlaps with 4 and the first of those
    auto columns = [&](int io, int k0, float (&w)[4], int &ks) {
        int n = 0;
        ks = 0;
        w[0] = w[1] = w[2] = w[3] = 0.f;
        if (io < no && cell) {
            const float c = cen(g.d_pix, io, no);
            const float cp = v.po * c, co = v.oo * c;
            const float2 sz = __ldg(tab + (size_t)ia * nm + io);
            const float a = fmaf(Ul, g.DSO - co, -g.DSD * cp) * rl * inv_d + 0.5f * nd;
            const float b = fmaf(Ur, g.DSO - co, -g.DSD * cp) * rr * inv_d + 0.5f * nd;
            const float fl = fminf(a, b), fh = fmaxf(a, b);
            ks = pole ? 0 : (int)floorf(fminf(fmaxf(fl, 0.f), (float)(nd - 1)));
            n = pole ? nd : fh >= 0.f && fl < (float)nd ? min((int)floorf(fh), nd - 1) - ks + 1 : 0;
            if (k0 > 0) ks = n > k0 ? ks + k0 : 0;
            float pa = projU(g, v, cp, co, edg(g.d_pix, ks, nd));
            const float sc = sz.x * sz.y * g.d_pix;  // v-overlaps are in slices
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float pb = projU(g, v, cp, co, edg(g.d_pix, ks + t + 1, nd));
                const float o = fminf(fmaxf(pa, pb), Ur) - fmaxf(fminf(pa, pb), Ul);
                w[t] = (k0 + t < n && o > 0.f) ? o * sc : 0.f;
                pa = pb;
            }
        }
        return n;
    };
    int ngrp = 0;
    for (int ib = 0; ib < no; ib += 4) {
        unsigned wide4, long4, live4;
        {
            const int io = ib + ls;
            float w[4];
            int ks;
            const int n = columns(io, 0, w, ks);
            bool fit = true, miss = false;
            if (cs == 0 && io < no) {
                const double b = __ldg(&bt[(size_t)ia * nm + io].y);
                const Line l = line_at(b, fma(b, vd, 0.5 * g.nz), zn);
                fit = l.fits<Strip<VEC, M>::NW>() && !big;
                miss = fit && (l.start + l.rows <= 0 || l.start >= g.nz);
                W.line[ls] = l.pack(rev, fit);
            }
            wide4 = __ballot_sync(0xffffffffu, n > 4 || (!WIDE && !fit));
            long4 = WIDE ? __ballot_sync(0xffffffffu, !fit) : 0;
            live4 = __ballot_sync(0xffffffffu, n > 0) & ~(__ballot_sync(0xffffffffu, miss) * 0xffu);
            put_column(W, ls, cs, w, ks, min(n, 4));
            __syncwarp();
        }
        const int nb = min(4, no - ib);
        for (int sv = 0; sv < nb; ++sv) {
            if (!(live4 >> (8 * sv) & 0xff)) continue;
            const int io = ib + sv;
            if (!WIDE && (wide4 >> (8 * sv) & 0xff)) {
                const float c = cen(g.d_pix, io, no);
                const float cp = v.po * c, co = v.oo * c;
                const float2 sz = __ldg(tab + (size_t)ia * nm + io);
#pragma unroll
                for (int j = 0; j < BT; ++j)
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const int iv = v0 + 32 * m + lane;
                        if (u0 + j < g.nu && iv < g.nv)
                            grp[j][m] += sz.x * fp_cell_line(g, v, vol, sk, so, nd, io, cp, co, sz.y,
                                                             ufloor_edge(g, u0 + j), ufloor_edge(g, u0 + j + 1),
                                                             vfloor_edge(g, iv), vfloor_edge(g, iv + 1));
                    }
            } else {
                // the next 4 pixels of the cells over more than k0
                auto more = [&](int k0) {
                    int n = 0;
                    if constexpr (WIDE) {
                        if (!(wide4 >> (8 * sv) & 0xff)) return false;
                        float w[4];
                        int ks;
                        n = columns(io, k0, w, ks);
                        __syncwarp();
                        put_column(W, sv, cs, w, ks, max(min(n - k0, 4), 0), ls == sv);
                        __syncwarp();
                    }
                    return WIDE && __any_sync(0xffffffffu, n > k0);
                };
                int k0 = 0;
                if (WIDE && (long4 >> (8 * sv) & 1)) {
                    do {
#pragma unroll
                        for (int c0 = 0; c0 < BT; c0 += 2) {
                            const LongPair<M> p = long_pair<M>(W, sv, c0, vol + io * so, sk, zn, g.nz);
#pragma unroll
                            for (int m = 0; m < M; ++m) {
                                grp[c0][m] += p.a[m];
                                grp[c0 + 1][m] += p.b[m];
                            }
                        }
                    } while (more(k0 += 4));
                } else {
                    do {
                        Strip<VEC, M> st;
                        st.init(vol + io * so, (unsigned)sk, lane, W.line[sv], zn, g.nz);
#pragma unroll
                        for (int c0 = 0; c0 < BT; c0 += 2) st.pair(W, sv, c0, lane, grp[c0], grp[c0 + 1]);
                    } while (more(k0 += 4));
                }
            }
            if (++ngrp == FP_GROUP) {
#pragma unroll
                for (int c = 0; c < BT; ++c)
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        acc[c * SZ + 32 * m] += grp[c][m];
                        grp[c][m] = 0.f;
                    }
                ngrp = 0;
            }
        }
        __syncwarp();  // the table and the row buffers are reused
    }
    const float f = g.d_pix * g.d_pix / (g.du * g.dv);
#pragma unroll
    for (int c = 0; c < BT; ++c)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int iv = v0 + 32 * m + lane;
            if (u0 + c < g.nu && iv < g.nv) {
                const size_t o = ((size_t)ia * g.nu + u0 + c) * g.nv + iv;
                float fp = (acc[c * SZ + 32 * m] + grp[c][m]) * f;
                if (MODE) {  // SIRT residual: (y - FP) / W_sino, FP kept where W_sino == 0
                    const float wi = inv_w[o];
                    fp = (wi != 0.f) ? (y[o] - fp) * wi : fp;
                }
                sino[o] = fp;
            }
        }
}

template <int MODE, int VEC, int M, bool WIDE>
int launch_fp_t(const vg_dd3d_geom *g, const float *vol, const Ws3 &w, float *sino, const float *y,
                const float *inv_w, cudaStream_t st) {
    constexpr size_t smem = FPW * (BT * 32 * M * sizeof(float) + sizeof(WarpBuf));
    int s = cuda_status(cudaFuncSetAttribute(dd3d_fp_kernel<MODE, VEC, M, WIDE>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                        "dd3d_fp");
    if (s) return s;
    dim3 grid(ceil_div(g->nv, 32 * M), ceil_div(g->nu, BT * FPW), g->na);
    dd3d_fp_kernel<MODE, VEC, M, WIDE><<<grid, 32 * FPW, smem, st>>>(*g, vol, w.vf, w.tab, w.bt, sino, y, inv_w);
    return launch_status("dd3d_fp");
}

template <int MODE, bool WIDE>
int launch_fp_w(const vg_dd3d_geom *g, const float *vol, const Ws3 &w, float *sino, const float *y,
                const float *inv_w, int M, cudaStream_t st) {
    const bool vec = g->nz % 4 == 0 && ((uintptr_t)vol & 15) == 0;
    switch (M) {
        case 3: return vec ? launch_fp_t<MODE, 4, 3, WIDE>(g, vol, w, sino, y, inv_w, st)
                           : launch_fp_t<MODE, 1, 3, WIDE>(g, vol, w, sino, y, inv_w, st);
        case 2: return vec ? launch_fp_t<MODE, 4, 2, WIDE>(g, vol, w, sino, y, inv_w, st)
                           : launch_fp_t<MODE, 1, 2, WIDE>(g, vol, w, sino, y, inv_w, st);
        default: return vec ? launch_fp_t<MODE, 4, 1, WIDE>(g, vol, w, sino, y, inv_w, st)
                            : launch_fp_t<MODE, 1, 1, WIDE>(g, vol, w, sino, y, inv_w, st);
    }
}

template <int MODE>
int launch_fp(const vg_dd3d_geom *g, const float *vol, const Ws3 &w, float *sino, const float *y,
              const float *inv_w, cudaStream_t st) {
    // 96 or 64 v cells per warp while the slices under them fit a column buffer,
    // by the smallest magnification a line of the volume can have; 96 unless the
    // detector's last tile is emptier for it
    const double r = 0.5 * hypot((double)g->nx, (double)g->ny) * g->d_pix;
    const double bmax = (g->DSO + r) / g->DSD * g->dv / g->d_pix;
    int M = 1;
    if (g->nv > 32 && 96.0 * bmax + 9.0 <= BW && 96 * ceil_div(g->nv, 96) <= 1.15 * 64 * ceil_div(g->nv, 64))
        M = 3;
    else if (g->nv > 32 && 64.0 * bmax + 9.0 <= BW)
        M = 2;
    // 32 where that leaves few blocks (200 of 64 v cells, 200^3 and 4 views: 0.33 ms, of
    // 32 cells 0.30; 288, 128^3 and 16 views: 0.221 against 0.228)
    if ((long long)ceil_div(g->nv, 32 * M) * ceil_div(g->nu, BT * FPW) * g->na < 250) M = 1;
    // WIDE from u cells of 3.2 pixels on, by the widest at the far side of the volume
    // (128^3, 120 views: 0.65 against 0.78 ms at 3.0, 1.44 against 0.77 at 3.4), and
    // where rows do not fit (v cells of 4 slices, 180 views: 3.8 against 2.4 ms)
    const bool wide = 32.0 * M * bmax + 9.0 > BW || 1.415 * (g->DSO + r) / g->DSD * g->du / g->d_pix > 3.2;
    return wide ? launch_fp_w<MODE, true>(g, vol, w, sino, y, inv_w, M, st)
                : launch_fp_w<MODE, false>(g, vol, w, sino, y, inv_w, M, st);
}

// Backprojection.  Block = 8 x 8 columns (x, y) x 32 M slices; a warp owns one
// pixel line of the tile (8 columns along the view's driving axis) and walks
// the views, 4 at a time.  Its warps wait for each other only where the
// driving axis changes and a voxel's sum moves to another warp.  Sums: 16
// views in registers, then a compensated sum per voxel in shared memory.
// Lines whose voxels cover more than 4 detector columns, or more rows than a column
// buffer holds, take the per-voxel global path; WIDE, where such columns are many and
// the rows fit, takes 4 columns at a time.  With too few tiles to
// fill the GPU, a cluster of up to 8 blocks shares a tile, each with a part of
// the views; their sums are added in rank order through distributed shared
// memory.  At 80 registers 3 blocks fit an SM (256^3: 9.3 ms; 2 blocks of 128
// registers, or 4 of 64 with spills, 11.4 / 11.3 ms).
__device__ float bp_voxel_view(const vg_dd3d_geom &g, const View3 &v, const float *__restrict__ s,
                               float2 sz, int k, int nd, float cp, float co, int iz) {
    const float u0 = ufloor_edge(g, 0), v0 = vfloor_edge(g, 0);
    const float idu = 1.0f / g.du, idv = 1.0f / g.dv;
    const float pa = projU(g, v, cp, co, edg(g.d_pix, k, nd));
    const float pb = projU(g, v, cp, co, edg(g.d_pix, k + 1, nd));
    const float ulo = fminf(pa, pb), uhi = fmaxf(pa, pb);
    const float vlo = sz.y * edg(g.d_pix, iz, g.nz), vhi = sz.y * edg(g.d_pix, iz + 1, g.nz);
    const int j0 = max(0, (int)floorf((ulo - u0) * idu)), j1 = min(g.nu - 1, (int)floorf((uhi - u0) * idu));
    const int q0 = max(0, (int)floorf((vlo - v0) * idv)), q1 = min(g.nv - 1, (int)floorf((vhi - v0) * idv));
    float part = 0.f;
    for (int j = j0; j <= j1; ++j) {
        const float ou = fminf(uhi, ufloor_edge(g, j + 1)) - fmaxf(ulo, ufloor_edge(g, j));
        if (ou <= 0.f) continue;
        float rs = 0.f;
        for (int q = q0; q <= q1; ++q) {
            const float ov = fminf(vhi, vfloor_edge(g, q + 1)) - fmaxf(vlo, vfloor_edge(g, q));
            if (ov > 0.f) rs = fmaf(__ldg(s + (size_t)j * g.nv + q), ov, rs);
        }
        part = fmaf(rs, ou, part);
    }
    return part * sz.x;
}

#ifndef VG_CONE_BP_MINB
#define VG_CONE_BP_MINB 3
#endif

// MODE 0: back projection; 1: SIRT update epilogue.  VEC: floats per sinogram
// load (4 needs nv % 4 == 0 and a 16-byte aligned sinogram).
template <int MODE, int VEC, int M, bool WIDE>
__global__ void __launch_bounds__(256, VG_CONE_BP_MINB)
dd3d_bp_kernel(vg_dd3d_geom g, const float *__restrict__ sino, const float4 *__restrict__ vf,
               const float2 *__restrict__ tab, const double2 *__restrict__ bt, float *__restrict__ vol,
               const float *__restrict__ inv_w, float gamma) {
    constexpr int SZ = 32 * M;
    extern __shared__ float4 smem4[];
    float2 *kh = reinterpret_cast<float2 *>(smem4);  // [BT * BT][SZ] (sum, compensation)
    cg::cluster_group cl = cg::this_cluster();
    const int S = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int z0 = (blockIdx.x / S) * SZ, y0 = blockIdx.y * BT, x0 = blockIdx.z * BT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    WarpBuf &W = reinterpret_cast<WarpBuf *>(kh + BT * BT * SZ)[warp];
    const int nm = g.nx > g.ny ? g.nx : g.ny;
    const float idu = 1.0f / g.du, u0 = ufloor_edge(g, 0);
    const int zn = min(SZ, g.nz - z0);
    const double zd = (double)(z0 + (zn >> 1)) - 0.5 * g.nz, cv = 0.5 * g.nv - (double)g.sv;  // the middle slice's edge
    for (int i = tid; i < BT * BT * SZ; i += 256) kh[i] = make_float2(0.f, 0.f);
    __syncthreads();
    float grp[BT][M];
#pragma unroll
    for (int c = 0; c < BT; ++c)
#pragma unroll
        for (int m = 0; m < M; ++m) grp[c][m] = 0.f;
    int ngrp = 0, axis = -1;
    auto flush = [&]() {
#pragma unroll
        for (int c = 0; c < BT; ++c) {
            float2 *k = kh + (axis ? c + BT * warp : warp + BT * c) * SZ + lane;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                Kahan a;
                a.s = k[32 * m].x; a.c = k[32 * m].y;
                a.add(grp[c][m]);
                k[32 * m] = make_float2(a.s, a.c);
                grp[c][m] = 0.f;
            }
        }
        ngrp = 0;
    };
    const int ls = lane >> 3, cs = lane & 7;
    // detector columns under voxel column cs of the warp's line in view ia: their number,
    // and from the k0-th on the overlaps with 4 and the first of those
    auto columns = [&](int ia, const View3 &v, int k0, float (&w)[4], int &js) {
        const int nd = v.xdrv ? g.nx : g.ny, no = v.xdrv ? g.ny : g.nx;
        const int k = (v.xdrv ? x0 : y0) + cs, io = (v.xdrv ? y0 : x0) + warp;
        int n = 0;
        js = 0;
        w[0] = w[1] = w[2] = w[3] = 0.f;
        if (io < no) {
            const float sc = __ldg(tab + (size_t)ia * nm + io).x * g.dv;
            const float ce = cen(g.d_pix, io, no);
            const float cp = v.po * ce, co = v.oo * ce;
            const float pa = projU(g, v, cp, co, edg(g.d_pix, k, nd));
            const float pb = projU(g, v, cp, co, edg(g.d_pix, k + 1, nd));
            const float ulo = fminf(pa, pb), uhi = fmaxf(pa, pb);
            js = max((int)floorf((ulo - u0) * idu), 0);
            n = k < nd ? max(min((int)floorf((uhi - u0) * idu), g.nu - 1) - js + 1, 0) : 0;
            js = min(js, g.nu - 1);
            if (k0 > 0) js = n > k0 ? js + k0 : 0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float o = fminf(uhi, ufloor_edge(g, js + t + 1)) - fmaxf(ulo, ufloor_edge(g, js + t));
                w[t] = (k0 + t < n && o > 0.f) ? o * sc : 0.f;
            }
        }
        return n;
    };
    const int va0 = (int)((long long)g.na * rank / S), va1 = (int)((long long)g.na * (rank + 1) / S);
    for (int ib = va0; ib < va1; ib += 4) {
        // u-overlaps of views ib .. ib + 3 (lane = view * 8 + column)
        unsigned xdrv4, wide4, live4;
        {
            const int ia = min(ib + ls, g.na - 1);
            const View3 v = view_f(vf, ia);
            float w[4];
            int js;
            const int n = columns(ia, v, 0, w, js);
            bool fit = true, miss = false;
            const int io = (v.xdrv ? y0 : x0) + warp;
            if (cs == 0 && io < (v.xdrv ? g.ny : g.nx)) {
                const double b = __ldg(&bt[(size_t)ia * nm + io].x);
                const Line l = line_at(b, fma(b, zd, cv), zn);
                fit = l.fits<Strip<VEC, M>::NW>();
                miss = fit && (l.start + l.rows <= 0 || l.start >= g.nv);
                W.line[ls] = l.pack(v.pd < 0.f, true);
            }
            xdrv4 = __ballot_sync(0xffffffffu, v.xdrv);
            wide4 = __ballot_sync(0xffffffffu, n > 4 || (!WIDE && !fit));
            live4 = __ballot_sync(0xffffffffu, n > 0) & ~(__ballot_sync(0xffffffffu, miss) * 0xffu);
            put_column(W, ls, cs ^ (int)(v.pd < 0.f), w, js, min(n, 4));
            __syncwarp();
        }
        const int nb = min(4, va1 - ib);
        for (int sv = 0; sv < nb; ++sv) {
            const int ia = ib + sv, xd = (xdrv4 >> (8 * sv)) & 1;
            if (xd != axis) {  // block-uniform: every warp walks the same views
                if (axis >= 0) {
                    flush();
                    __syncthreads();
                }
                axis = xd;
            }
            const bool live = (live4 >> (8 * sv)) & 0xff;
            if (live) {
                const float *s = sino + (size_t)ia * g.nu * g.nv;
                if (!WIDE && (wide4 >> (8 * sv) & 0xff)) {
                    const View3 v = view_f(vf, ia);
                    const int nd = v.xdrv ? g.nx : g.ny, no = v.xdrv ? g.ny : g.nx;
                    const int io = (v.xdrv ? y0 : x0) + warp;
                    const float ce = cen(g.d_pix, io, no);
#pragma unroll
                    for (int c = 0; c < BT; ++c)
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            const int k = (v.xdrv ? x0 : y0) + c, iz = z0 + 32 * m + lane;
                            if (k < nd && iz < g.nz)
                                grp[c][m] += bp_voxel_view(g, v, s, __ldg(tab + (size_t)ia * nm + io),
                                                           k, nd, v.po * ce, v.oo * ce, iz);
                        }
                } else {
                    // the next 4 detector columns of the voxels over more than k0
                    auto more = [&](int k0) {
                        int n = 0;
                        if constexpr (WIDE) {
                            if (!(wide4 >> (8 * sv) & 0xff)) return false;
                            const View3 v = view_f(vf, ia);
                            float w[4];
                            int js;
                            n = columns(ia, v, k0, w, js);
                            __syncwarp();
                            put_column(W, sv, cs ^ (int)(v.pd < 0.f), w, js, max(min(n - k0, 4), 0), ls == sv);
                            __syncwarp();
                        }
                        return WIDE && __any_sync(0xffffffffu, n > k0);
                    };
                    int k0 = 0;
                    do {
                        Strip<VEC, M> st;
                        st.init(s, g.nv, lane, W.line[sv], zn, g.nv);
#pragma unroll
                        for (int c0 = 0; c0 < BT; c0 += 2) st.pair(W, sv, c0, lane, grp[c0], grp[c0 + 1]);
                    } while (more(k0 += 4));
                }
            }
            if (++ngrp == BP_GROUP) flush();
        }
        __syncwarp();  // the table and the row buffers are reused
    }
    if (axis >= 0) flush();
    const float f = 1.0f / ((float)g.na * g.d_pix);
    if (S > 1) cl.sync();
    else __syncthreads();
    // rows of the tile, split over the cluster's blocks
    for (int col = warp * S + rank; col < BT * BT; col += 8 * S) {
        const int ix = x0 + (col & 7), iy = y0 + (col >> 3);
        if (ix >= g.nx || iy >= g.ny) continue;
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
                    const float2 q = *cl.map_shared_rank(k, r);
                    a.merge(q);
                }
            }
            const size_t o = ((size_t)ix * g.ny + iy) * g.nz + z0 + iz;
            const float bp = a.s * f;
            if (MODE) {  // SIRT update: x += gamma BP / W_img, BP where W_img == 0
                const float wi = inv_w[o];
                vol[o] += gamma * ((wi != 0.f) ? bp * wi : bp);
            } else {
                vol[o] = bp;
            }
        }
    }
    if (S > 1) cl.sync();  // no block leaves while its sums are read
}

// Blocks of a cluster that share a tile: until every SM has about three blocks, 16
// views per block at least (360 views, until one, three and six blocks: 64^3 0.223,
// 0.237 and 0.237 ms, 96^3 0.78, 0.85 and 0.72, 128^3 1.50, 1.50 and 1.25).
int bp_split(const vg_dd3d_geom *g, long long tiles) {
    int S = 1;
    while (S < 8 && tiles * S < 3 * NSM && g->na >= 32 * S) S *= 2;
    return S;
}

constexpr size_t bp_smem(int M) { return (size_t)BT * BT * 32 * M * sizeof(float2) + 8 * sizeof(WarpBuf); }

template <int MODE, int VEC, int M, bool WIDE>
int launch_bp_t(const vg_dd3d_geom *g, const float *sino, const Ws3 &w, float *vol, const float *inv_w, float gamma, cudaStream_t st) {
    const long long tiles = (long long)ceil_div(g->nz, 32 * M) * ceil_div(g->ny, BT) * ceil_div(g->nx, BT);
    const int S = bp_split(g, tiles);
    int s = cuda_status(cudaFuncSetAttribute(dd3d_bp_kernel<MODE, VEC, M, WIDE>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)bp_smem(M)), "dd3d_bp");
    if (s) return s;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(ceil_div(g->nz, 32 * M) * S, ceil_div(g->ny, BT), ceil_div(g->nx, BT));
    c.blockDim = dim3(256);
    c.dynamicSmemBytes = bp_smem(M);
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&c, dd3d_bp_kernel<MODE, VEC, M, WIDE>, *g, sino, w.vf, w.tab, w.bt, vol,
                                          inv_w, gamma), "dd3d_bp");
}

template <int MODE, bool WIDE>
int launch_bp_w(const vg_dd3d_geom *g, const float *sino, const Ws3 &w, float *vol, const float *inv_w,
                float gamma, bool two, cudaStream_t st) {
    const bool vec = g->nv % 4 == 0 && ((uintptr_t)sino & 15) == 0;
    if (two) return vec ? launch_bp_t<MODE, 4, 2, WIDE>(g, sino, w, vol, inv_w, gamma, st)
                        : launch_bp_t<MODE, 1, 2, WIDE>(g, sino, w, vol, inv_w, gamma, st);
    return vec ? launch_bp_t<MODE, 4, 1, WIDE>(g, sino, w, vol, inv_w, gamma, st)
               : launch_bp_t<MODE, 1, 1, WIDE>(g, sino, w, vol, inv_w, gamma, st);
}

template <int MODE>
int launch_bp(const vg_dd3d_geom *g, const float *sino, const Ws3 &w, float *vol, const float *inv_w,
              float gamma, cudaStream_t st) {
    // 64 slices per warp while the rows they project to fit a column buffer, by the
    // largest magnification a line of the volume can have -- also where the last tile is
    // then emptier (96 x 96 x 65, 300 views: 0.70 ms, with 32 0.77) -- and there are
    // about as many blocks as SMs (64^3, 8 views: 64 blocks 28.7 us, 128 of 32 slices 24.6)
    const double r = 0.5 * hypot((double)g->nx, (double)g->ny) * g->d_pix;
    const double mag = g->DSD / (g->DSO - fmin(r, 0.999 * g->DSO)), bmax = mag * g->d_pix / g->dv;
    const long long tiles = (long long)ceil_div(g->nz, 64) * ceil_div(g->ny, BT) * ceil_div(g->nx, BT);
    const bool two = g->nz > 32 && 64.0 * bmax + 9.0 <= BW && tiles * bp_split(g, tiles) >= 100;
    // WIDE from voxels of 4.6 detector columns on, by the widest at the near side (128^3,
    // 120 views: 0.57 against 0.62 ms at 4.4, 1.12 against 0.73 at 5.4).  Where rows do
    // not fit the per-voxel path is the faster (slices over 4 v cells, 180 views: 3.8
    // against 4.9 ms by long_pair, with voxels over 4 columns too 4.6 against 5.8)
    const bool fit = two || 32.0 * bmax + 9.0 <= BW;  // then so on every line
    const bool wide = fit && 1.415 * mag * g->d_pix / g->du > 4.6;
    return wide ? launch_bp_w<MODE, true>(g, sino, w, vol, inv_w, gamma, two, st)
                : launch_bp_w<MODE, false>(g, sino, w, vol, inv_w, gamma, two, st);
}

int check(const vg_dd3d_geom *g) {
    VG_REQUIRE(g, "dd3d: null geometry");
    VG_REQUIRE(g->nx > 0 && g->ny > 0 && g->nz > 0 && g->na > 0 && g->nu > 0 && g->nv > 0,
               "dd3d: sizes must be positive");
    VG_REQUIRE(g->na < 65536 && g->nx < 65536 && ceil_div(g->nu, 8) < 65536 &&
                   ceil_div(g->ny, 8) < 65536, "dd3d: sizes too large for the grid");
    VG_REQUIRE(g->du > 0.f && g->dv > 0.f && g->d_pix > 0.f && g->DSO > 0.f && g->DSD > 0.f,
               "dd3d: pitches and distances must be positive");
    const float h = 0.5f * (float)(g->nx > g->ny ? g->nx : g->ny) * g->d_pix;
    VG_REQUIRE(h < 0.70710678f * g->DSO, "dd3d: volume half-width must be below DSO/sqrt(2)");
    return VG_OK;
}

int launch_prep(const vg_dd3d_geom *g, const double *trig, void *ws, size_t wsb, cudaStream_t st) {
    VG_REQUIRE(ws && wsb >= ws_bytes(g) && ((uintptr_t)ws & 15) == 0,
               "dd3d: workspace of %zu bytes needed (vg_dd3d_workspace_bytes)", ws_bytes(g));
    const Ws3 w = ws_of(g, ws);
    dd3d_prep<<<g->na, 256, 0, st>>>(*g, trig, const_cast<float2 *>(w.tab), const_cast<float4 *>(w.vf),
                                     const_cast<double2 *>(w.bt));
    return launch_status("dd3d_prep");
}

}  // namespace

extern "C" size_t vg_dd3d_workspace_bytes(const vg_dd3d_geom *g) {
    return check(g) ? 0 : ws_bytes(g);
}

extern "C" int vg_dd3d_fp(const vg_dd3d_geom *g, const float *vol, const double *trig,
                          float *sino, void *workspace, size_t workspace_bytes, void *stream) {
    int s = check(g);
    if (s) return s;
    VG_REQUIRE(vol && trig && sino, "dd3d_fp: null pointer");
    cudaStream_t st = as_stream(stream);
    s = launch_prep(g, trig, workspace, workspace_bytes, st);
    if (s) return s;
    return launch_fp<0>(g, vol, ws_of(g, workspace), sino, nullptr, nullptr, st);
}

extern "C" int vg_dd3d_bp(const vg_dd3d_geom *g, const float *sino, const double *trig,
                          float *vol, void *workspace, size_t workspace_bytes, void *stream) {
    int s = check(g);
    if (s) return s;
    VG_REQUIRE(vol && trig && sino, "dd3d_bp: null pointer");
    cudaStream_t st = as_stream(stream);
    s = launch_prep(g, trig, workspace, workspace_bytes, st);
    if (s) return s;
    return launch_bp<0>(g, sino, ws_of(g, workspace), vol, nullptr, 0.f, st);
}

extern "C" int vg_dd3d_sirt_iter(const vg_dd3d_geom *g, const float *y, const float *inv_w_sino,
                                 const float *inv_w_img, float gamma, const double *trig, float *x,
                                 float *r, void *workspace, size_t workspace_bytes, void *stream) {
    int s = check(g);
    if (s) return s;
    VG_REQUIRE(y && inv_w_sino && inv_w_img && trig && x && r, "dd3d_sirt_iter: null pointer");
    cudaStream_t st = as_stream(stream);
    s = launch_prep(g, trig, workspace, workspace_bytes, st);
    if (s) return s;
    const Ws3 w = ws_of(g, workspace);
    s = launch_fp<1>(g, x, w, r, y, inv_w_sino, st);
    if (s) return s;
    return launch_bp<1>(g, r, w, x, inv_w_img, gamma, st);
}
