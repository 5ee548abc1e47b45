// Pixel-driven FBP backprojection (parallel and flat-detector fan).
//
// After ramp filtering (filtration.filter_sino, which applies 2H), the
// reconstruction of a full scan (pi parallel or 2 pi either geometry) is
//     f(x, y) = pi / (2 na) * sum_views Q(s(x, y)) / U(x, y)^2
// with, in vir's distance-driven geometry (source direction (cos, sin),
// detector axis (-sin, cos), dd.py:486-494, 527-585):
//     o = cos x + sin y,  p = -sin x + cos y,
//     parallel: s = p, U = 1;
//     fan:      s = DSD p / (DSO - o) on the detector, U = (DSO - o) / DSO,
// Q linearly interpolated between bin centres du (j - nu/2 + 0.5 + su) and
// zero outside the detector.  The fan weights are the equispaced
// (collinear-detector) ones whose pre-weight is the reference's
// cosine_weighting(equispaced=True) (processing/reconstruction.py:99-107) and
// whose distance weight is the 1/U^2 of its Hsieh backprojector
// (processing/proj2.py:606-613).
#include <cooperative_groups.h>

#include "vg_common.cuh"

namespace {

using namespace vg;
namespace cg = cooperative_groups;

// Thread = PX pixels of a column strip (x0 + 8 i, y), lanes along y.  What
// bounded the plain form (one pixel per thread, (cos, sin) read and converted
// from FP64 by every thread and view) was the FP64 pipe: two conversions per
// warp and view at 2 lanes per clock took 0.64 of its 0.69 ms at 512 x 512, 720
// views.  The block now converts its views once, VB at a time, into shared
// memory: 0.19 ms, bound by instruction issue (78 %, 29 per pixel and view; 1 or
// 4 pixels per thread are 14 and 3 % slower).  A cluster of S blocks shares a tile when the tiles alone would not
// fill the GPU, each block with a part of the views; their compensated sums are
// added in rank order through distributed shared memory.
constexpr int PX = 2, VB = 256;

template <bool FAN>
__global__ void __launch_bounds__(256)
fbp2d_bp_kernel(vg_dd2d_geom g, const float *__restrict__ q, const double *__restrict__ trig, float scale,
                float *__restrict__ img) {
    __shared__ float2 view[VB];        // (cos, sin)
    __shared__ float2 part[PX][256];   // (sum, compensation) of this block's views
    cg::cluster_group cl = cg::this_cluster();
    const int S = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int iy = (blockIdx.x / S) * 32 + threadIdx.x;
    const int ix = blockIdx.y * 8 * PX + threadIdx.y;
    float x[PX];
#pragma unroll
    for (int i = 0; i < PX; ++i) x[i] = g.d_pix * ((float)(ix + 8 * i) + 0.5f - 0.5f * g.nx);
    const float y = g.d_pix * ((float)iy + 0.5f - 0.5f * g.ny);
    // s -> bins: counted from the bin at the detector's middle, so that the
    // rounding of the coordinate is that of half the detector
    const float k = FAN ? __fdiv_rn(g.DSD, g.du) : __fdiv_rn(1.0f, g.du);
    const float off = 0.5f * g.nu - 0.5f - g.su, mid = floorf(off), fo = off - mid;
    const int jm = (int)mid;
    const int va0 = (int)((long long)g.na * rank / S), va1 = (int)((long long)g.na * (rank + 1) / S);
    // per-view terms summed in groups of 16 views, the group sums compensated
    Kahan acc[PX];
    float grp[PX];
#pragma unroll
    for (int i = 0; i < PX; ++i) grp[i] = 0.f;
    for (int vb = va0; vb < va1; vb += VB) {
        const int nb = min(VB, va1 - vb);
        __syncthreads();
        if (tid < nb) {
            view[tid] = make_float2((float)__ldg(trig + 2 * (vb + tid)), (float)__ldg(trig + 2 * (vb + tid) + 1));
        }
        __syncthreads();
        const float *row = q + (size_t)vb * g.nu;
#pragma unroll 4
        for (int v = 0; v < nb; ++v, row += g.nu) {
            const float2 cs = view[v];
            const float py = cs.x * y, dy = fmaf(-cs.y, y, g.DSO);
#pragma unroll
            for (int i = 0; i < PX; ++i) {
                float p = fmaf(-cs.y, x[i], py), w = 1.0f;
                if (FAN) {
                    const float r = recip_n(fmaf(-cs.x, x[i], dy));
                    p *= r;
                    w = (g.DSO * r) * (g.DSO * r);  // 1 / U^2
                }
                const float t = fmaf(p, k, fo), ft = floorf(t);
                const int j = (int)ft + jm;
                const float v0 = (unsigned)j < (unsigned)g.nu ? __ldg(row + j) : 0.f;
                const float v1 = (unsigned)(j + 1) < (unsigned)g.nu ? __ldg(row + j + 1) : 0.f;
                grp[i] = fmaf(w, fmaf(t - ft, v1 - v0, v0), grp[i]);
            }
            if ((v & 15) == 15) {
#pragma unroll
                for (int i = 0; i < PX; ++i) {
                    acc[i].add(grp[i]);
                    grp[i] = 0.f;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < PX; ++i) {
        acc[i].add(grp[i]);
        if (S > 1) part[i][tid] = make_float2(acc[i].s, acc[i].c);
    }
    if (S > 1) {
        cl.sync();
        if (rank == 0) {
#pragma unroll
            for (int i = 0; i < PX; ++i)
                for (int r = 1; r < S; ++r) {
                    const float2 a = *cl.map_shared_rank(&part[i][tid], r);
                    acc[i].merge(a);
                }
        }
        cl.sync();  // no block leaves while its sums are read
        if (rank) return;
    }
#pragma unroll
    for (int i = 0; i < PX; ++i)
        if (ix + 8 * i < g.nx && iy < g.ny) img[(size_t)(ix + 8 * i) * g.ny + iy] = acc[i].s * scale;
}

template <bool FAN>
int launch(const vg_dd2d_geom *g, const float *q, const double *trig, float scale, float *img,
           cudaStream_t st) {
    const int tx = ceil_div(g->ny, 32), ty = ceil_div(g->nx, 8 * PX);
    // blocks until every SM has eight (2048 threads), 16 views per block at least (512 x
    // 512, 720 views, filter included: until four 0.265 ms, eight 0.246, sixteen 0.251)
    int S = 1;
    while (S < 8 && (long long)tx * ty * S < 8 * NSM && g->na >= 32 * S) S *= 2;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(tx * S, ty);
    c.blockDim = dim3(32, 8);
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&c, fbp2d_bp_kernel<FAN>, *g, q, trig, scale, img), "fbp2d_bp");
}

}  // namespace

extern "C" int vg_fbp2d_bp(const vg_dd2d_geom *g, const float *q, const double *trig, float *img,
                           void *stream) {
    VG_REQUIRE(g && q && trig && img, "fbp2d_bp: null pointer");
    VG_REQUIRE(g->nx > 0 && g->ny > 0 && g->na > 0 && g->nu > 0, "fbp2d_bp: bad sizes");
    VG_REQUIRE(g->du > 0.f && g->d_pix > 0.f, "fbp2d_bp: du and d_pix must be positive");
    VG_REQUIRE(!g->fan || (g->DSO > 0.f && g->DSD > 0.f), "fbp2d_bp: fan needs DSO, DSD > 0");
    VG_REQUIRE(ceil_div(g->nx, 8) < 65536, "fbp2d_bp: nx too large");
    const float scale = (float)(3.14159265358979323846 / (2.0 * g->na));
    return g->fan ? launch<true>(g, q, trig, scale, img, as_stream(stream))
                  : launch<false>(g, q, trig, scale, img, as_stream(stream));
}
