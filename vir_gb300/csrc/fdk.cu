// FDK (Feldkamp-Davis-Kress) reconstruction for the circular cone-beam
// geometry of dd_fp_cone_3d: cosine pre-weight, row ramp filter along u,
// distance-weighted voxel-driven backprojection.
//
// vir has no FDK; the weights extend its fan-beam specification to
// the cone: the equispaced pre-weight of processing/reconstruction.py:99-107
// becomes DSD / sqrt(DSD^2 + u^2 + v^2) on the flat detector, the filter is
// filtration.filter_sino's 2H at the isocentre pitch du DSO / DSD, and the
// backprojection carries the 1/U^2 weight of processing/proj2.py:606-613:
//     f(x, y, z) = pi / (2 na) sum_views Q(u, v) / U^2,
//     o = c x + s y, p = -s x + c y, U = (DSO - o) / DSO,
//     u = DSD p / (DSO - o), v = DSD z / (DSO - o),
// with Q bilinearly interpolated between bin centres (zero outside).
#include "vg_common.cuh"

namespace {

using namespace vg;

// (na, nu, nv) -> weighted (na, nv, nu)
__global__ void fdk_weight_transpose(vg_dd3d_geom g, const float *__restrict__ in,
                                     float *__restrict__ out) {
    __shared__ float tile[32][33];
    const int ia = blockIdx.z;
    const int v0 = blockIdx.x * 32, u0 = blockIdx.y * 32;
    const float *src = in + (size_t)ia * g.nu * g.nv;
    float *dst = out + (size_t)ia * g.nu * g.nv;
    for (int q = threadIdx.y; q < 32; q += blockDim.y) {
        const int iu = u0 + q, iv = v0 + threadIdx.x;
        if (iu < g.nu && iv < g.nv) {
            const float u = g.du * ((float)iu - 0.5f * g.nu + 0.5f + g.su);
            const float v = g.dv * ((float)iv - 0.5f * g.nv + 0.5f + g.sv);
            const float w = g.DSD * rsqrtf(g.DSD * g.DSD + u * u + v * v);
            tile[q][threadIdx.x] = src[(size_t)iu * g.nv + iv] * w;
        }
    }
    __syncthreads();
    for (int q = threadIdx.y; q < 32; q += blockDim.y) {
        const int iv = v0 + q, iu = u0 + threadIdx.x;
        if (iu < g.nu && iv < g.nv) dst[(size_t)iv * g.nu + iu] = tile[threadIdx.x][q];
    }
}

// (na, nv, nu) -> (na, nu, nv)
__global__ void fdk_transpose_back(vg_dd3d_geom g, const float *__restrict__ in,
                                   float *__restrict__ out) {
    __shared__ float tile[32][33];
    const int ia = blockIdx.z;
    const int u0 = blockIdx.x * 32, v0 = blockIdx.y * 32;
    const float *src = in + (size_t)ia * g.nu * g.nv;
    float *dst = out + (size_t)ia * g.nu * g.nv;
    for (int q = threadIdx.y; q < 32; q += blockDim.y) {
        const int iv = v0 + q, iu = u0 + threadIdx.x;
        if (iu < g.nu && iv < g.nv) tile[q][threadIdx.x] = src[(size_t)iv * g.nu + iu];
    }
    __syncthreads();
    for (int q = threadIdx.y; q < 32; q += blockDim.y) {
        const int iu = u0 + q, iv = v0 + threadIdx.x;
        if (iu < g.nu && iv < g.nv) dst[(size_t)iu * g.nv + iv] = tile[threadIdx.x][q];
    }
}

// Warp = one (x, y) column, 64 H of its slices: lane + 32 t, t < 2 H, so that
// each tap load covers about 32 neighbouring rows of one detector column.
//
// All that a view needs of the column (u, 1 / U, the v step, whether every tap
// lies on the detector) is the same in every lane, so the lanes work it out
// for 32 views at a time, one view each, into a table; a view then costs one
// broadcast read, and a voxel without a tap off the detector runs no branch:
// the loads of all its slices are issued together.  A column partly off the
// detector takes view_edges, tap by tap.
//
// Bound by L1: a tap load is about two wavefronts, a voxel eight cycles of an
// SM (L1 86 % busy; issue 58 %).  Against threads of four consecutive slices
// with the view's terms, the detector test and 64-bit addresses per thread (34
// instructions a voxel, now 22): 512^3, 720 views of 1024 x 768, FDK 147.8 ->
// 109 ms, the results the same bits.  Four blocks of eight warps (64
// registers): with five the loads of a view no longer fit (129 ms), with three
// too few are in flight (132 ms); columns in 2 x 8, 4 x 4, 2 x 4 blocks 112, 111,
// 111 ms.
struct FdkView {
    float au, w, zr;
    int off;  // first tap's row offset ju nv; EDGES or NONE
};
constexpr int FDK_EDGES = -1;  // some tap may lie off the detector
constexpr int FDK_NONE = -2;   // every tap does

// Whether the n floats at p have one high address word.
__device__ __forceinline__ bool one_page(const float *p, int n) {
    return (reinterpret_cast<unsigned long long>(p) >> 32) ==
           (reinterpret_cast<unsigned long long>(p + n) >> 32);
}

__device__ __forceinline__ FdkView fdk_view(const vg_dd3d_geom &g, const float *Qa, float2 t2, float x,
                                            float y, float z0, float z1) {
    const float iu_off = 0.5f * g.nu - 0.5f - g.su, iv_off = 0.5f * g.nv - 0.5f - g.sv;
    const float idu = 1.0f / g.du, idv = 1.0f / g.dv;
    const float c = t2.x, s = t2.y;
    const float d = g.DSO - fmaf(c, x, s * y);
    const float r = 1.0f / d;
    const float p = fmaf(-s, x, c * y);
    const float tu = g.DSD * p * r * idu + iu_off;
    const float fu = floorf(tu);
    const float Ui = g.DSO * r;  // 1 / U
    FdkView v;
    v.au = tu - fu;
    v.w = Ui * Ui;
    v.zr = g.DSD * r * idv;
    // the slices' v lie between those of the first and the last
    const float va = fmaf(z0, v.zr, iv_off), vb = fmaf(z1, v.zr, iv_off);
    const bool in = fu >= 0.f && fu < (float)(g.nu - 1) && fminf(va, vb) >= 0.f &&
                    fmaxf(va, vb) < (float)(g.nv - 1) && g.nv <= (1 << 22) &&
                    (long long)g.nu * g.nv <= 0x7fffffffLL && one_page(Qa + (long long)fu * g.nv, 2 * g.nv);
    const bool none = (fu < -1.f || fu >= (float)g.nu) && v.w < INFINITY;
    v.off = in ? (int)fu * g.nv : none ? FDK_NONE : FDK_EDGES;
    return v;
}

// One view of a column whose taps may lie off the detector, where they are 0.
template <int H>
__device__ __forceinline__ void view_edges(const vg_dd3d_geom &g, const float *Qa, float2 t2, float x,
                                           float y, const float2 (&z)[H], float2 (&grp)[H]) {
    const float iu_off = 0.5f * g.nu - 0.5f - g.su, iv_off = 0.5f * g.nv - 0.5f - g.sv;
    const FdkView v = fdk_view(g, Qa, t2, x, y, 0.f, 0.f);
    const float r = 1.0f / (g.DSO - fmaf(t2.x, x, t2.y * y));
    const float p = fmaf(-t2.y, x, t2.x * y);
    const int ju = (int)floorf(g.DSD * p * r * (1.0f / g.du) + iu_off);
    auto at = [&](int j, int k) -> float {
        return (j >= 0 && j < g.nu && k >= 0 && k < g.nv) ? __ldg(Qa + (size_t)j * g.nv + k) : 0.f;
    };
    auto term = [&](float z, float grp) -> float {
        const float tv = fmaf(z, v.zr, iv_off);
        const float fv = floorf(tv);
        const int jv = (int)fv;
        const float av = tv - fv;
        const float q00 = at(ju, jv), q01 = at(ju, jv + 1);
        const float q10 = at(ju + 1, jv), q11 = at(ju + 1, jv + 1);
        const float a = fmaf(av, q01 - q00, q00), b = fmaf(av, q11 - q10, q10);
        return fmaf(fmaf(v.au, b - a, a), v.w, grp);
    };
#pragma unroll
    for (int h = 0; h < H; ++h) grp[h] = make_float2(term(z[h].x, grp[h].x), term(z[h].y, grp[h].y));
}

constexpr int FDK_COLS = 8;  // columns of a block, consecutive in y
template <int H>
__global__ void __launch_bounds__(32 * FDK_COLS, 4)
fdk_bp_kernel(vg_dd3d_geom g, const float *__restrict__ q, const double *__restrict__ trig,
              float scale, float *__restrict__ vol) {
    __shared__ float4 tab[FDK_COLS][32];   // FdkView of 32 views, per warp
    extern __shared__ float2 cs[];  // (cos, sin) per view
    for (int ia = threadIdx.y * 32 + threadIdx.x; ia < g.na; ia += 32 * FDK_COLS)
        cs[ia] = make_float2((float)__ldg(trig + 2 * ia), (float)__ldg(trig + 2 * ia + 1));
    __syncthreads();
    const int lane = threadIdx.x, zb = blockIdx.x * 64 * H;
    const int iy = blockIdx.y * FDK_COLS + threadIdx.y;
    const int ix = blockIdx.z;
    if (iy >= g.ny) return;
    const float x = g.d_pix * ((float)ix + 0.5f - 0.5f * g.nx);
    const float y = g.d_pix * ((float)iy + 0.5f - 0.5f * g.ny);
    // slices past the last repeat it and are not stored
    auto zat = [&](int iz) { return g.d_pix * ((float)min(iz, g.nz - 1) + 0.5f - 0.5f * g.nz); };
    float2 z[H];
#pragma unroll
    for (int h = 0; h < H; ++h) z[h] = make_float2(zat(zb + lane + 64 * h), zat(zb + lane + 64 * h + 32));
    const float z0 = zat(zb), z1 = zat(zb + 64 * H - 1);
    const float iv_off = 0.5f * g.nv - 0.5f - g.sv;
    const size_t plane = (size_t)g.nu * g.nv;
    // per-view terms summed in groups of 16 views, the group sums compensated
    Kahan acc[2 * H];
    for (int ib = 0; ib < g.na; ib += 16) {
        if ((ib & 31) == 0) {
            __syncwarp();
            const int il = min(ib + lane, g.na - 1);
            const FdkView v = fdk_view(g, q + il * plane, cs[il], x, y, z0, z1);
            tab[threadIdx.y][lane] = make_float4(v.au, v.w, v.zr, __int_as_float(v.off));
            __syncwarp();
        }
        float2 grp[H];
#pragma unroll
        for (int h = 0; h < H; ++h) grp[h] = dup(0.f);
        const int ie = min(ib + 16, g.na);
        for (int ia = ib; ia < ie; ++ia) {
            const float4 v = tab[threadIdx.y][ia & 31];
            const int off = __float_as_int(v.w);
            const float *Qa = q + ia * plane;
            if (off < 0) {
                if (off == FDK_EDGES) view_edges(g, Qa, cs[ia], x, y, z, grp);
                continue;
            }
            // addresses as 32-bit sums under the high word that all taps share
            const unsigned long long Q = reinterpret_cast<unsigned long long>(Qa + off);
            const unsigned hi = (unsigned)(Q >> 32), lo0 = (unsigned)Q - 0x2c000000u,
                           lo1 = lo0 + 4u * (unsigned)g.nv;
            auto tap = [hi](unsigned lo) {
                const float *p;
                asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "r"(lo), "r"(hi));
                return p;
            };
            float2 q00[H], q01[H], q10[H], q11[H], av[H];  // two slices each
#pragma unroll
            for (int h = 0; h < H; ++h) {
                // floor of tv in [0, 2^22): the sum's bits are those of 2^23 + floor
                const float2 tv = pk_fma(z[h], dup(v.z), dup(iv_off));
                const float2 b = pk_add_rd(tv, dup(8388608.f));
                av[h] = pk_sub(tv, pk_add(b, dup(-8388608.f)));
                // 0x2c000000 + 4 floor
                const unsigned jx = __float_as_uint(b.x) << 2, jy = __float_as_uint(b.y) << 2;
                const float *p0 = tap(lo0 + jx), *p1 = tap(lo1 + jx);
                const float *p2 = tap(lo0 + jy), *p3 = tap(lo1 + jy);
                q00[h] = make_float2(__ldg(p0), __ldg(p2));
                q01[h] = make_float2(__ldg(p0 + 1), __ldg(p2 + 1));
                q10[h] = make_float2(__ldg(p1), __ldg(p3));
                q11[h] = make_float2(__ldg(p1 + 1), __ldg(p3 + 1));
            }
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const float2 a = pk_fma(av[h], pk_sub(q01[h], q00[h]), q00[h]);
                const float2 b = pk_fma(av[h], pk_sub(q11[h], q10[h]), q10[h]);
                grp[h] = pk_fma(pk_fma(dup(v.x), pk_sub(b, a), a), dup(v.y), grp[h]);
            }
        }
#pragma unroll
        for (int h = 0; h < H; ++h) {
            acc[2 * h].add(grp[h].x);
            acc[2 * h + 1].add(grp[h].y);
        }
    }
    if ((g.na & 15) == 0)
#pragma unroll
        for (int t = 0; t < 2 * H; ++t) acc[t].add(0.f);  // folds in the compensation
#pragma unroll
    for (int t = 0; t < 2 * H; ++t) {
        const int iz = zb + lane + 32 * t;
        if (iz < g.nz) vol[((size_t)ix * g.ny + iy) * g.nz + iz] = acc[t].s * scale;
    }
}

template <int H>
int fdk_bp_launch(const vg_dd3d_geom *g, const float *q, const double *trig, float *vol, void *stream) {
    const float scale = (float)(3.14159265358979323846 / (2.0 * g->na));
    const size_t smem = (size_t)g->na * sizeof(float2);
    constexpr size_t limit = 200 * 1024;
    VG_REQUIRE(smem <= limit, "fdk_bp: more than 25600 views");
    if (smem > 40 * 1024) {  // to one limit for all sizes: other threads launch this kernel with theirs
        cudaError_t e = cudaFuncSetAttribute(fdk_bp_kernel<H>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
        if (e != cudaSuccess) return cuda_status(e, "fdk_bp: shared memory attribute");
    }
    dim3 grid(ceil_div(g->nz, 64 * H), ceil_div(g->ny, FDK_COLS), g->nx);
    fdk_bp_kernel<H><<<grid, dim3(32, FDK_COLS), smem, as_stream(stream)>>>(*g, q, trig, scale, vol);
    return launch_status("fdk_bp");
}

int check(const vg_dd3d_geom *g) {
    VG_REQUIRE(g && g->nx > 0 && g->ny > 0 && g->nz > 0 && g->na > 0 && g->nu > 0 && g->nv > 0,
               "fdk: sizes must be positive");
    VG_REQUIRE(g->nx < 65536 && g->na < 65536 && ceil_div(g->ny, 8) < 65536 &&
                   ceil_div(g->nu, 32) < 65536, "fdk: sizes too large");
    VG_REQUIRE(g->du > 0.f && g->dv > 0.f && g->d_pix > 0.f && g->DSO > 0.f && g->DSD > 0.f,
               "fdk: pitches and distances must be positive");
    return VG_OK;
}

}  // namespace

extern "C" int vg_fdk_weight_transpose(const vg_dd3d_geom *g, const float *sino, float *out,
                                       void *stream) {
    int s = check(g);
    if (s) return s;
    VG_REQUIRE(sino && out, "fdk_weight_transpose: null pointer");
    dim3 grid(ceil_div(g->nv, 32), ceil_div(g->nu, 32), g->na);
    fdk_weight_transpose<<<grid, dim3(32, 8), 0, as_stream(stream)>>>(*g, sino, out);
    return launch_status("fdk_weight_transpose");
}

extern "C" int vg_fdk_transpose_back(const vg_dd3d_geom *g, const float *in, float *out,
                                     void *stream) {
    int s = check(g);
    if (s) return s;
    VG_REQUIRE(in && out, "fdk_transpose_back: null pointer");
    dim3 grid(ceil_div(g->nu, 32), ceil_div(g->nv, 32), g->na);
    fdk_transpose_back<<<grid, dim3(32, 8), 0, as_stream(stream)>>>(*g, in, out);
    return launch_status("fdk_transpose_back");
}

extern "C" int vg_fdk_bp(const vg_dd3d_geom *g, const float *q, const double *trig, float *vol,
                         void *stream) {
    int s = check(g);
    if (s) return s;
    VG_REQUIRE(q && trig && vol, "fdk_bp: null pointer");
    // pairs of slices per lane: a view costs a warp about a quarter of a pair's
    // work besides its pairs', padded ones included (128 x 128 columns, 180 views, filter
    // included: 64 slices by one pair 0.34 ms, by two 0.40; 70: 0.52, 0.42; 128: 0.61,
    // 0.51; 200: 1.08, 0.87; at 129 to 192 and 257 to 320 slices, where the estimate takes
    // one, two would be 4 to 10 % faster: 140: 0.81, 0.78; 260: 1.35, 1.22)
    auto cost = [&](int h) { return (1 + 4 * h) * ceil_div(g->nz, 64 * h); };
    return cost(2) <= cost(1) ? fdk_bp_launch<2>(g, q, trig, vol, stream)
                              : fdk_bp_launch<1>(g, q, trig, vol, stream);
}
