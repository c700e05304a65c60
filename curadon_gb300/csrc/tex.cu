// tex.cu -- projection kernels that filter through the texture unit.
//
// The texture unit interpolates with 9-bit fixed-point weights (8 fractional
// bits), the same hardware path the reference samples through
// (texture.hpp:81-87: linear filtering, border address mode, unnormalised
// coordinates), so these variants reproduce the reference's interpolation
// exactly; the launch shapes, the single launch over all views and the
// resident arrays are this project's.
//
//  k_fwd2d_tex    2D forward, tex2D on a 2D array refreshed per call
//  k_bwd2d_tex    2D backprojection, tex1DLayered on the sinogram rows
//  k_fwd3d_tex3   3D forward, tex3D (trilinear in the texture unit)
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace cg {

// ------------------------------------------------------------ objects

int make_texture(cudaArray_t arr, cudaTextureObject_t *tex) {
    cudaResourceDesc res;
    std::memset(&res, 0, sizeof(res));
    res.resType = cudaResourceTypeArray;
    res.res.array.array = arr;
    cudaTextureDesc td;
    std::memset(&td, 0, sizeof(td));
    td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeBorder;
    td.filterMode = cudaFilterModeLinear;
    td.readMode = cudaReadModeElementType;
    td.normalizedCoords = 0;
    CG_TRY_CUDA(cudaCreateTextureObject(tex, &res, &td, nullptr));
    return CG_OK;
}

static int alloc_array(cudaArray_t *arr, size_t w, size_t h, size_t d, unsigned flags) {
    cudaChannelFormatDesc ch = cudaCreateChannelDesc<float>();
    CG_TRY_CUDA(cudaMalloc3DArray(arr, &ch, make_cudaExtent(w, h, d), flags));
    return CG_OK;
}

// Copies a dense (depth x height x width) float block into an array.
static int copy_to_array(cudaArray_t arr, const float *src, size_t w, size_t h, size_t d,
                         cudaStream_t s) {
    cudaMemcpy3DParms p;
    std::memset(&p, 0, sizeof(p));
    p.srcPtr = make_cudaPitchedPtr((void *)src, w * sizeof(float), w, h);
    p.dstArray = arr;
    p.extent = make_cudaExtent(w, h, d);
    p.kind = cudaMemcpyDeviceToDevice;
    CG_TRY_CUDA(cudaMemcpy3DAsync(&p, s));
    return CG_OK;
}

namespace {

// ------------------------------------------------------------ 2D forward

// The 32 x 32 tile (bx, by) of a volume into its texture's array.  A kernel of
// ours instead of a copy: the copy engine's hand-over costs more than the move
// of a small image (with launch_after, 64^2 x 360 views 10.2 -> 6.0 us a call in a
// CUDA graph, 12.3 -> 6.3 outside one), and a batch moves all its volumes in one
// launch.
template <class T>
__device__ __forceinline__ void fill_tile(cudaSurfaceObject_t surf, const T *__restrict__ vol,
                                          int W, int H, int bx, int by) {
    const int x = bx * 32 + (threadIdx.x & 31);
    if (x >= W) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int y = by * 32 + 8 * i + (threadIdx.x >> 5);
        if (y < H) surf2Dwrite(to_float(vol[(size_t)y * W + x]), surf, x * (int)sizeof(float), y);
    }
}

template <class T>
__global__ void __launch_bounds__(256)
    k_fill_tex(cudaSurfaceObject_t surf, const T *__restrict__ vol, int W, int H) {
    wait_previous();
    fill_tile(surf, vol, W, H, blockIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(256)
    k_batch_fill_tex(const Prob2d *__restrict__ probs, const int *__restrict__ start, int count) {
    wait_previous();
    const int i = batch_problem(start, count, blockIdx.x);
    const Prob2d &q = probs[i];
    const int lin = blockIdx.x - start[i], gx = (q.W + 31) / 32;
    fill_tile(q.surf, q.vol, q.W, q.H, lin % gx, lin / gx);
}

// Ray (u, view) of the reference's 2D forward (forward_2d.hpp:21-79) through
// the texture unit: its first sample, step and count; false where it misses.
struct TexRay {
    float x, y, vx, vy;
    int n;
};

__device__ __forceinline__ bool tex_ray(const float2 *__restrict__ tsrc,
                                        const float2 *__restrict__ tu0,
                                        const float2 *__restrict__ tdu, int W, int H, int u,
                                        int view, TexRay &r) {
    const float2 s = tsrc[view], o = tu0[view], du = tdu[view];
    const float fu = (float)u;
    const float dx = fmaf(du.x, fu, o.x);
    const float dy = fmaf(du.y, fu, o.y);
    float tmin = FLT_MIN, tmax = FLT_MAX;
    {
        const float t1 = __fdividef(-1.f - s.x, dx), t2 = __fdividef((float)W - s.x, dx);
        tmin = fminf(fmaxf(t1, tmin), fmaxf(t2, tmin));
        tmax = fmaxf(fminf(t1, tmax), fminf(t2, tmax));
    }
    {
        const float t1 = __fdividef(-1.f - s.y, dy), t2 = __fdividef((float)H - s.y, dy);
        tmin = fminf(fmaxf(t1, tmin), fmaxf(t2, tmin));
        tmax = fmaxf(fminf(t1, tmax), fminf(t2, tmax));
    }
    if ((double)tmin > (double)tmax - 1e-6) return false;
    r.x = fmaf(dx, tmin, s.x), r.y = fmaf(dy, tmin, s.y);
    const float tl = tmax - tmin;
    const float rdx = dx * tl, rdy = dy * tl;
    const float m = fmaxf(fabsf(rdx), fabsf(rdy));
    r.n = __float2int_rn(m);
    r.vx = rdx / m, r.vy = rdy / m;
    return true;
}

// The rays of a tile of kTexCells cells x 8 views, one warp per view: lane g *
// kTexCells + c takes run g of cell c's samples, kTexRuns runs of ceil(n /
// kTexRuns), stepping to its first one (the running sum of the positions, as
// the others make it); the runs' sums are added in pairs.  Against one lane per
// ray, four times the warps: small problems fill the SMs, the last round of
// blocks of the large ones is shorter, and a warp's 8 adjacent rays read a
// compact piece of the image at each of 4 places.  Bound by the texture unit's
// filtering (3.5 samples a clock and SM) from about 400^2 pixels, below by
// latency.  One lane per ray / this, us in a CUDA graph with the copy into the
// array: 64^2 x 360 views 12.3 / 10.2, 256^2 x 256 36.9 / 27.8, 512^2 x 512 160.6
// / 135.6, 640^2 x 100 78 / 57, 700^2 x 700 363 / 313; runs on adjacent lanes
// (adjacent lanes far apart in the image) 700^2 x 700 884; 8 cells x 4 views
// per warp without runs 358; 2 or 8 runs 327, 323.
constexpr int kTexRuns = 4, kTexCells = 8;

__device__ __forceinline__ void fwd2d_tex_tile(cudaTextureObject_t tex, float *__restrict__ sino,
                                               const float2 *__restrict__ tsrc,
                                               const float2 *__restrict__ tu0,
                                               const float2 *__restrict__ tdu, int W, int H,
                                               int det, int nangles, float sx, float sy, int bx,
                                               int by) {
    static_assert(kTexRuns * kTexCells == 32, "a warp per view");
    const int lane = threadIdx.x & 31, g = lane / kTexCells;
    const int u = bx * kTexCells + lane % kTexCells, view = by * 8 + (threadIdx.x >> 5);
    TexRay r;
    const bool hit = u < det && view < nangles && tex_ray(tsrc, tu0, tdu, W, H, u, view, r);
    float sum = 0.f;
    wait_previous();  // (the rays come from the plan's tables)
    if (hit) {
        const int run = (r.n + kTexRuns - 1) / kTexRuns;
        for (int j = 0; j < g * run; ++j) r.x += r.vx, r.y += r.vy;
        const int count = min(run, r.n - g * run);
#pragma unroll 4
        for (int j = 0; j < count; ++j) {
            sum += tex2D<float>(tex, r.x, r.y);
            r.x += r.vx;
            r.y += r.vy;
        }
    }
    // (every lane stays for the sums)
#pragma unroll
    for (int o = kTexCells; o < 32; o *= 2) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (g == 0 && u < det && view < nangles)
        sino[(size_t)view * det + u] = hit ? sum * hypotf(r.vx * sx, r.vy * sy) : 0.f;
}

__global__ void __launch_bounds__(256)
    k_fwd2d_tex(cudaTextureObject_t tex, float *__restrict__ sino,
                const float2 *__restrict__ tsrc, const float2 *__restrict__ tu0,
                const float2 *__restrict__ tdu, int W, int H, int det, int nangles, float sx,
                float sy) {
    fwd2d_tex_tile(tex, sino, tsrc, tu0, tdu, W, H, det, nangles, sx, sy, blockIdx.x, blockIdx.y);
}

// Many problems' texture forwards in one launch: the tiles of a (problem, tile)
// work list, each problem with its own texture (bindless handles in the work
// list).
__global__ void __launch_bounds__(256)
    k_batch_fwd2d_tex(const Prob2d *__restrict__ probs, const int *__restrict__ start,
                      int count) {
    const int i = batch_problem(start, count, blockIdx.x);
    const Prob2d &q = probs[i];
    const int t = blockIdx.x - start[i], tiles_u = (q.det + kTexCells - 1) / kTexCells;
    fwd2d_tex_tile(q.tex, q.sino, q.src, q.u0, q.du, q.W, q.H, q.det, q.nangles, q.sx, q.sy,
                   t % tiles_u, t / tiles_u);
}

// ------------------------------------------------------------ 2D backward

constexpr int kTexBwdRows = 4;
constexpr int kTexBwdViews = 256;

__global__ void __launch_bounds__(256)
    k_bwd2d_tex(float *__restrict__ vol, cudaTextureObject_t tex, const float4 *__restrict__ meta,
                int W, int H, int det, int v0, int nv, float sx, float sy, float ox, float oy,
                float ds, int ybase) {
    __shared__ float4 smeta[kTexBwdViews];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y0 = ybase + blockIdx.y * 32 + threadIdx.y;
    const float ex = (float)W / 2.0f, ey = (float)H / 2.0f, ed = (float)det / 2.0f;
    const float inv = __fdividef(1.0f, ds);
    const float X = ((float)x - ex) * sx + ox + 0.5f;
    const float SX = X * inv;
    float Y[kTexBwdRows], SY[kTexBwdRows], acc[kTexBwdRows];
#pragma unroll
    for (int r = 0; r < kTexBwdRows; ++r) {
        Y[r] = ((float)(y0 + 8 * r) - ey) * sy + oy + 0.5f;
        SY[r] = Y[r] * inv;
        acc[r] = 0.f;
    }
    for (int s0 = 0; s0 < nv; s0 += kTexBwdViews) {
        const int cnt = min(kTexBwdViews, nv - s0);
        __syncthreads();
        for (int i = tid; i < cnt; i += 256) smeta[i] = meta[v0 + s0 + i];
        __syncthreads();
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const float4 m = smeta[j];
            const float layer = (float)(s0 + j);
#pragma unroll
            for (int r = 0; r < kTexBwdRows; ++r) {
                const float xi = m.x * X - m.y * Y[r];
                const float yi = m.y * SX + m.x * SY[r];
                const float w = __fdividef(m.z, xi + m.w);
                const float u = w * yi + ed;
                acc[r] = fmaf(tex1DLayered<float>(tex, u, (int)layer), w, acc[r]);
            }
        }
    }
    if (x < W) {
#pragma unroll
        for (int r = 0; r < kTexBwdRows; ++r) {
            const int y = y0 + 8 * r;
            if (y < H) vol[(size_t)y * W + x] += acc[r] * inv;
        }
    }
}

// ------------------------------------------------------------ 3D forward

struct RaySeg {
    float sx, sy, sz, dx, dy, dz, tmin, tmax, h;
    int nsteps;
    bool hit;
};

// Ray set-up of forward_3d.hpp:56-81 (intersection.h:12-28).
__device__ __forceinline__ RaySeg ray3d(const float4 o, const float4 du, const float4 dv,
                                        const float4 s, int iu, int iv, int X, int Y, int Z) {
    RaySeg r;
    const float fu = (float)iu, fv = (float)iv;
    const float detx = o.x + fu * du.x + fv * dv.x;
    const float dety = o.y + fu * du.y + fv * dv.y;
    const float detz = o.z + fu * du.z + fv * dv.z;
    r.sx = s.x, r.sy = s.y, r.sz = s.z;
    r.dx = detx - s.x, r.dy = dety - s.y, r.dz = detz - s.z;
    const float len = sqrtf(r.dx * r.dx + r.dy * r.dy + r.dz * r.dz);
    const long long nsamples = (long long)ceilf(__fdividef(len, 1.0f));
    float tmin = FLT_MIN, tmax = FLT_MAX;
    {
        const float t1 = __fdividef(-1.f - s.x, r.dx), t2 = __fdividef((float)(X + 1) - s.x, r.dx);
        tmin = fminf(fmaxf(t1, tmin), fmaxf(t2, tmin));
        tmax = fmaxf(fminf(t1, tmax), fminf(t2, tmax));
    }
    {
        const float t1 = __fdividef(-1.f - s.y, r.dy), t2 = __fdividef((float)(Y + 1) - s.y, r.dy);
        tmin = fminf(fmaxf(t1, tmin), fmaxf(t2, tmin));
        tmax = fmaxf(fminf(t1, tmax), fminf(t2, tmax));
    }
    {
        const float t1 = __fdividef(-1.f - s.z, r.dz), t2 = __fdividef((float)(Z + 1) - s.z, r.dz);
        tmin = fminf(fmaxf(t1, tmin), fmaxf(t2, tmin));
        tmax = fmaxf(fminf(t1, tmax), fminf(t2, tmax));
    }
    r.tmin = tmin, r.tmax = tmax;
    r.hit = tmin <= tmax;
    r.nsteps = r.hit ? (int)ceilf((tmax - tmin) * (float)nsamples) : 0;
    r.h = r.hit ? (tmax - tmin) / (float)r.nsteps : 0.f;
    if (!(r.h > 0.f) || !isfinite(tmax) || r.nsteps > (1 << 22)) r.hit = false;
    return r;
}

__global__ void __launch_bounds__(256)
    k_fwd3d_tex3(cudaTextureObject_t tex, float *__restrict__ sino,
                 const float4 *__restrict__ torg, const float4 *__restrict__ tdu,
                 const float4 *__restrict__ tdv, const float4 *__restrict__ tsrc, int X, int Y,
                 int Z, int U, int V, int P, bool exact_t) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.y * blockDim.y + threadIdx.y;
    const int view = blockIdx.z * blockDim.z + threadIdx.z;
    if (iu >= U || iv >= V || view >= P) return;
    const RaySeg r = ray3d(torg[view], tdu[view], tdv[view], tsrc[view], iu, iv, X, Y, Z);
    if (!r.hit) return;
    float acc = 0.f, t = r.tmin;
    for (int k = 0; k <= r.nsteps + 1; ++k) {
        if (!(t <= r.tmax)) break;
        acc += tex3D<float>(tex, fmaf(r.dx, t, r.sx) + 0.5f, fmaf(r.dy, t, r.sy) + 0.5f,
                            fmaf(r.dz, t, r.sz) + 0.5f);
        t = march_next(t, k, r.tmin, r.h, exact_t);
    }
    sino[((size_t)view * V + iv) * U + iu] = acc;
}

}  // namespace

// ------------------------------------------------------------ launchers

int tex_blocks(const Plan2d &p) { return ceil_div(p.det, kTexCells) * ceil_div(p.nangles, 8); }

int launch_forward2d_tex(Plan2d &p, const void *vol, bool half, float *sino, cudaStream_t s) {
    if (int rc = ensure_vol_texture(p)) return rc;
    const dim3 grid(ceil_div(p.det, kTexCells), ceil_div(p.nangles, 8));
    if (grid.y > 65535) return set_error(CG_ERR_INVALID, "too many views for one launch");
    auto fill = [&](auto kernel, auto *from) {
        return launch_after(kernel, dim3(ceil_div(p.W, 32), ceil_div(p.H, 32)), 256, 0, s, 1,
                            p.surf_vol, from, p.W, p.H);
    };
    if (int rc = half ? fill(k_fill_tex<__half>, static_cast<const __half *>(vol))
                      : fill(k_fill_tex<float>, static_cast<const float *>(vol)))
        return rc;
    return launch_after(k_fwd2d_tex, grid, 256, 0, s, 1, p.tex_vol, sino, p.d_src, p.d_u0, p.d_du,
                        p.W, p.H, p.det, p.nangles, p.sx, p.sy);
}

int ensure_vol_texture(Plan2d &p) {
    int rc = CG_OK;
    if (!p.arr_vol && (rc = alloc_array(&p.arr_vol, p.W, p.H, 0, cudaArraySurfaceLoadStore)))
        return rc;
    if (!p.surf_vol) {
        cudaResourceDesc res;
        std::memset(&res, 0, sizeof(res));
        res.resType = cudaResourceTypeArray;
        res.res.array.array = p.arr_vol;
        CG_TRY_CUDA(cudaCreateSurfaceObject(&p.surf_vol, &res));
    }
    if (!p.tex_vol) return make_texture(p.arr_vol, &p.tex_vol);
    return CG_OK;
}

int launch_batch2d_fwd_tex(const Prob2d *probs, const int *starts, const int totals[kBatchStages],
                           int count, int fill, int rays, cudaStream_t s) {
    if (totals[rays] == 0) return CG_OK;
    if (int rc = launch_after(k_batch_fill_tex, totals[fill], 256, 0, s, 1, probs,
                              starts + fill * (count + 1), count))
        return rc;
    return launch_after(k_batch_fwd2d_tex, totals[rays], 256, 0, s, 1, probs,
                        starts + rays * (count + 1), count);
}

int launch_backward2d_tex(Plan2d &p, float *vol, const float *sino, cudaStream_t s) {
    constexpr int kLayers = 2048;  // layered 1D arrays hold at most 2048 layers
    if (!p.arr_sino) {
        const int layers = std::min(p.nangles, kLayers);
        int rc = alloc_array(&p.arr_sino, p.det, 0, layers, cudaArrayLayered);
        if (rc) return rc;
        if ((rc = make_texture(p.arr_sino, &p.tex_sino))) return rc;
    }
    dim3 grid(ceil_div(p.W, 32), ceil_div(p.H, 32));
    for (int v0 = 0; v0 < p.nangles; v0 += kLayers) {
        const int nv = std::min(kLayers, p.nangles - v0);
        int rc = copy_to_array(p.arr_sino, sino + (size_t)v0 * p.det, p.det, 1, nv, s);
        if (rc) return rc;
        k_bwd2d_tex<<<grid, dim3(32, 8), 0, s>>>(vol, p.tex_sino, p.d_bmeta, p.W, p.H, p.det, v0,
                                                 nv, p.sx, p.sy, p.ox, p.oy, p.ds, 0);
        CG_TRY_CUDA(cudaGetLastError());
    }
    return CG_OK;
}

int ensure_volume_texture3(Plan3d &p) {
    if (!p.arr3) {
        int rc = alloc_array(&p.arr3, p.X, p.Y, p.Z, cudaArrayDefault);
        if (rc) return rc;
        if ((rc = make_texture(p.arr3, &p.tex3))) return rc;
    }
    return CG_OK;
}

int upload_volume_texture3(Plan3d &p, const float *vol, cudaStream_t s) {
    if (int rc = ensure_volume_texture3(p)) return rc;
    return copy_to_array(p.arr3, vol, p.X, p.Y, p.Z, s);
}

int launch_forward3d_tex(Plan3d &p, const float *vol, float *sino, cudaStream_t s) {
    const dim3 block(p.fwd_bx, p.fwd_by, p.fwd_bz);
    const dim3 grid(ceil_div(p.U, p.fwd_bx), ceil_div(p.V, p.fwd_by), ceil_div(p.nangles, p.fwd_bz));
    if (grid.z > 65535) return set_error(CG_ERR_INVALID, "too many views for one launch");
    int rc = upload_volume_texture3(p, vol, s);
    if (rc) return rc;
    k_fwd3d_tex3<<<grid, block, 0, s>>>(p.tex3, sino, p.d_forg, p.d_fdu, p.d_fdv, p.d_fsrc, p.X,
                                        p.Y, p.Z, p.U, p.V, p.nangles, p.exact_t);
    CG_TRY_CUDA(cudaGetLastError());
    return CG_OK;
}

}  // namespace cg
