// Post-processing: left-right check with nearest-neighbour plane fill,
// colour-weighted median over planes, plane -> disparity, and the single-pair
// driver's 7-tap separable median. Reference: PostProcess (post_process.cu:
// 4-185, :373-390; CPU/OpenMP there) and medianFilter
// (main_stereo_hbp_isp.cu:120-192).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "engine.h"

namespace hbp
{
namespace
{
__device__ __forceinline__ float get_z(const float *v, int x, int y)
{
    return v[0] * (float)x + v[1] * (float)y + v[2];
}

// doConsistencyCheck (post_process.cu:4-41), left view: fail where the right
// disparity at int(x - d + 0.5f) differs by more than 1.5.
__global__ void lr_fail_kernel(const float *dispL, const float *dispR, int W, int H, uint8_t *fail)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H)
        return;
    int y = i / W, x = i - y * W;
    float ds = dispL[i];
    uint8_t f = 0;
    if (ds == ds)
    {
        int rx = (int)((float)x - ds * 1.0f + 0.5f);
        if (rx >= 0 && rx < W && fabsf(dispR[y * W + rx] - ds) > 1.5f)
            f = 255;
    }
    fail[i] = f;
}

// cv::dilate with a 3x3 box; samples outside the image do not take part.
__global__ void dilate3_kernel(const uint8_t *in, int W, int H, uint8_t *out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H)
        return;
    int y = i / W, x = i - y * W;
    uint8_t m = 0;
    for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx)
        {
            int yy = y + dy, xx = x + dx;
            if (yy >= 0 && yy < H && xx >= 0 && xx < W)
                m = max(m, in[yy * W + xx]);
        }
    out[i] = m;
}

// Horizontal NN-interpolation (post_process.cu:72-109): nearest pixel on
// each side outside the dilated mask; keep the plane with the smaller
// disparity at the failed pixel. Reads only pixels outside the dilated mask,
// writes only failed pixels (a subset of it), so the update is in place.
__global__ void lr_fill_kernel(const uint8_t *fail, const uint8_t *fail2, int W, int H, float *plane)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H || !fail[i])
        return;
    int y = i / W, x = i - y * W;
    int xl = x, xr = x;
    while (xl >= 0 && fail2[y * W + xl] == 255)
        xl--;
    while (xr < W && fail2[y * W + xr] == 255)
        xr++;
    const float *pl = xl >= 0 ? plane + 3 * (size_t)(y * W + xl) : nullptr;
    const float *pr = xr < W ? plane + 3 * (size_t)(y * W + xr) : nullptr;
    const float *pick;
    if (!pl && !pr)
        return;
    else if (!pl)
        pick = pr;
    else if (!pr)
        pick = pl;
    else
        pick = get_z(pl, x, y) < get_z(pr, x, y) ? pl : pr;
    float a = pick[0], b = pick[1], c = pick[2];
    plane[3 * (size_t)i] = a;
    plane[3 * (size_t)i + 1] = b;
    plane[3 * (size_t)i + 2] = c;
}

__global__ void plane_to_disp_kernel(const float *plane, int W, int H, float *disp)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H)
        return;
    int y = i / W, x = i - y * W;
    disp[i] = get_z(plane + 3 * (size_t)i, x, y);
}

// What the weighted median reads of a pixel in one 16-byte load: its plane
// (x, y, z) and its colour's three bytes (the bits of w). The failed pixels'
// list is taken on the way.
__global__ void pack_and_list(const uint8_t *bgr, const uint8_t *fail, const float *plane, int n, float4 *px, int *list,
                              int *count)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = i < n;
    if (in)
    {
        const float *pl = plane + 3 * (size_t)i;
        const uint8_t *c = bgr + 3 * (size_t)i;
        px[i] = make_float4(pl[0], pl[1], pl[2], __uint_as_float(c[0] | (uint32_t)c[1] << 8 | (uint32_t)c[2] << 16));
    }
    const bool f = in && fail[i];
    const unsigned m = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && m)
        base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (f)
        list[base + __popc(m & ((1u << lane) - 1u))] = i;
}

// sum|dBGR| of two packed colours
__device__ __forceinline__ int colour_dist(float a, float b)
{
    return (int)__dp4a(__vabsdiffu4(__float_as_uint(a), __float_as_uint(b)), 0x01010101u, 0u);
}
// a packed pixel's plane at (x, y)
__device__ __forceinline__ float get_z(float4 v, float x, float y) { return v.x * x + v.y * y + v.z; }

// Weighted median (post_process.cu:127-185) of the pixels that
// weighted_select_kernel leaves over: one block per pixel, its window sorted.
// Window samples (41x41 clipped) get weight expf(-sum|dBGR| / 10) and the
// disparity of their plane at the pixel; the samples are sorted by
// (disparity, window position) and the first one whose cumulative weight
// exceeds half the total gives the plane. Weight sums are in double. A NaN
// disparity counts as +infinity (the reference's std::sort has no order for
// it), and so does the padding, which its index keeps behind every sample: the
// first n sorted entries are the window's.
// The colour distance sum|dBGR| is an integer 0..765, so the weights come
// from a 766-entry table computed on the host with the C library's expf,
// the function the reference's CPU code calls.
constexpr int WM_T = 256, WM_N = 2048, WM_R = 20;
__global__ void __launch_bounds__(WM_T)
    weighted_median_kernel(const float4 *px, const int *list, const int *count, int W, int H, float *plane,
                           const float *wtab)
{
    __shared__ float zk[WM_N];
    __shared__ int ik[WM_N];
    __shared__ double part[WM_T];
    __shared__ int found, close;
    for (int item = blockIdx.x; item < *count; item += gridDim.x)
    {
        __syncthreads(); // the previous pixel is done with the shared arrays
        const int p = list[item];
        const int y = p / W, x = p - y * W;
        const int y0 = max(y - WM_R, 0), y1 = min(y + WM_R + 1, H);
        const int x0 = max(x - WM_R, 0), x1 = min(x + WM_R + 1, W);
        const int ww = x1 - x0, n = ww * (y1 - y0);
        const float colour = px[p].w;
        for (int j = threadIdx.x; j < WM_N; j += WM_T)
        {
            if (j < n)
            {
                int q = (y0 + j / ww) * W + x0 + j % ww;
                const float z = get_z(px[q], (float)x, (float)y);
                zk[j] = z == z ? z : INFINITY;
                ik[j] = j;
            }
            else
            {
                zk[j] = INFINITY;
                ik[j] = WM_N + j;
            }
        }
        __syncthreads();
        // bitonic sort by (z, index)
        for (int k = 2; k <= WM_N; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1)
            {
                for (int t = threadIdx.x; t < WM_N; t += WM_T)
                {
                    int u = t ^ j;
                    if (u > t)
                    {
                        bool up = (t & k) == 0;
                        float za = zk[t], zb = zk[u];
                        int ia = ik[t], ib = ik[u];
                        bool gt = za > zb || (za == zb && ia > ib);
                        if (gt == up)
                        {
                            zk[t] = zb;
                            zk[u] = za;
                            ik[t] = ib;
                            ik[u] = ia;
                        }
                    }
                }
                __syncthreads();
            }
        // weights in sorted order; block prefix sums in double (fixed order)
        const int per = WM_N / WM_T; // 8 consecutive sorted samples per thread
        double wv[per];
        double tsum = 0.0;
        for (int k = 0; k < per; ++k)
        {
            int j = threadIdx.x * per + k;
            double w = 0.0;
            if (j < n)
            {
                int src = ik[j];
                int q = (y0 + src / ww) * W + x0 + src % ww;
                w = (double)wtab[colour_dist(colour, px[q].w)];
            }
            wv[k] = w;
            tsum += w;
        }
        part[threadIdx.x] = tsum;
        if (threadIdx.x == 0)
        {
            found = 0x7fffffff;
            close = 0;
        }
        __syncthreads();
        // inclusive scan of per-thread sums (Hillis-Steele, fixed order)
        for (int off = 1; off < WM_T; off <<= 1)
        {
            double v = threadIdx.x >= off ? part[threadIdx.x - off] : 0.0;
            __syncthreads();
            part[threadIdx.x] += v;
            __syncthreads();
        }
        const double center = part[WM_T - 1] / 2.0;
        double run = threadIdx.x ? part[threadIdx.x - 1] : 0.0, before = 0.0;
        int mine = 0x7fffffff;
        for (int k = 0; k < per; ++k)
        {
            int j = threadIdx.x * per + k;
            before = run;
            run += wv[k];
            if (j < n && run > center)
            {
                mine = j;
                atomicMin(&found, j);
                break;
            }
        }
        // the crossing sample when rounding cannot move it; otherwise the sums
        // are taken one by one, the total in window order and the running
        // weight in sorted order, as the reference does
        const double eps = 1e-11 * center;
        __syncthreads();
        if (found < n && mine == found && (run - center <= eps || center - before <= eps))
            close = 1;
        __syncthreads();
        if (close)
        {
            for (int k = 0; k < per; ++k)
                if (threadIdx.x * per + k < n)
                    zk[ik[threadIdx.x * per + k]] = (float)wv[k]; // weights by window position
            __syncthreads();
            if (threadIdx.x == 0)
            {
                double total = 0.0, sum = 0.0;
                for (int j = 0; j < n; ++j)
                    total += (double)zk[j];
                found = 0x7fffffff;
                for (int j = 0; j < n && found == 0x7fffffff; ++j)
                {
                    sum += (double)zk[ik[j]];
                    if (sum > total / 2.0)
                        found = j;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && found < n)
        {
            int src = ik[found];
            int q = (y0 + src / ww) * W + x0 + src % ww;
            plane[3 * (size_t)p] = px[q].x;
            plane[3 * (size_t)p + 1] = px[q].y;
            plane[3 * (size_t)p + 2] = px[q].z;
        }
    }
}

// PostProcess::median_filter_gpu (post_process.cu:188-371), the reference's
// GPU variant of the weighted median, for the pixels that
// weighted_select_kernel leaves over: one warp per pixel. Window samples in
// row-major order get the device patch weight wtab[sum|dBGR|]
// (expf(-k / 10), launch_patch_weights) and z = fma(a, x, b * y) + c, the
// reference device code's evaluation of a * x + b * y + c; the total weight
// is a float sum in window order. The reference orders the samples with
// bubble_sort (:216-229): step i swaps into position i, in scan order, every
// later sample smaller than the current one there. Its effect is a rotation
// along the chain of strict running minima of [i, n): position i takes the
// last of the chain, each chain member the previous one's sample, the first
// member the old sample at i; position i is then final. Each step cuts
// [i+1, n) into 32 contiguous chunks (an odd chunk length keeps the lanes in
// distinct shared-memory banks), finds the running minimum before each chunk
// by an ordered scan of the chunk minima, reads the samples the chain hands
// on across chunk borders, then lets each lane walk its chunk carrying the
// previous chain member's sample. The running weight in float stops the sort
// at the first sample past half the total, whose plane is taken. NaN
// disparities never enter a chain, as NaN compares false there.
constexpr int WG_MAXN = (2 * WM_R + 1) * (2 * WM_R + 1); // window samples (1681)
constexpr int WG_W = 2;                                    // pixels (warps) per block

// the earlier of two (z, pos) candidates unless the later is strictly smaller;
// pos < 0: none
__device__ __forceinline__ void first_min(float &z, int &p, float z2, int p2)
{
    if (p2 >= 0 && (p < 0 || z2 < z))
    {
        z = z2;
        p = p2;
    }
}

__global__ void __launch_bounds__(32 * WG_W)
    weighted_median_gpu_kernel(const float4 *__restrict__ px, const int *__restrict__ list,
                               const int *__restrict__ count, int W, int H, float *__restrict__ plane,
                               const float *__restrict__ wtab)
{
    __shared__ float zs_all[WG_W][WG_MAXN], ws_all[WG_W][WG_MAXN];
    __shared__ int ids_all[WG_W][WG_MAXN];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *zs = zs_all[wid], *ws = ws_all[wid];
    int *ids = ids_all[wid];
    for (int item = blockIdx.x * WG_W + wid; item < *count; item += gridDim.x * WG_W) // warp-uniform
    {
        __syncwarp(); // the previous pixel is done with the shared arrays
        const int p = list[item];
        const int y = p / W, x = p - y * W;
        const int y0 = max(y - WM_R, 0), y1 = min(y + WM_R, H - 1);
        const int x0 = max(x - WM_R, 0), x1 = min(x + WM_R, W - 1);
        const int ww = x1 - x0 + 1, n = ww * (y1 - y0 + 1);
        const float colour = px[p].w;
        const float fx = (float)x, fy = (float)y;
        for (int j = lane; j < n; j += 32)
        {
            const float4 v = px[(size_t)(y0 + j / ww) * W + x0 + j % ww];
            ws[j] = wtab[colour_dist(colour, v.w)];
            zs[j] = __fadd_rn(__fmaf_rn(v.x, fx, __fmul_rn(v.y, fy)), v.z);
            ids[j] = j;
        }
        __syncwarp();
        float center = 0.f;
        if (lane == 0)
        {
            float sum = 0.f;
            for (int j = 0; j < n; ++j)
                sum = __fadd_rn(sum, ws[j]);
            center = __fdiv_rn(sum, 2.0f);
        }
        float run = 0.f; // lane 0's running weight in sorted order
        int pick = -1;
        for (int i = 0; i < n; ++i)
        {
            const float zi = zs[i];
            const bool chain = zi == zi; // a NaN at i is never displaced
            const int m = n - i - 1;
            const int c = ((m + 31) >> 5) | 1;
            const int lo = min(i + 1 + lane * c, n), hi = min(lo + c, n);
            // the chunk's first minimum (NaN samples never qualify)
            float cz = 0.f;
            int cp = -1;
            for (int j = lo; j < hi; ++j)
            {
                const float zj = zs[j];
                if (zj == zj)
                    first_min(cz, cp, zj, j);
            }
            // ordered inclusive scan of the chunk minima over the lanes
            float sz = cz;
            int sp = cp;
    #pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                const float oz = __shfl_up_sync(0xffffffffu, sz, off);
                const int op = __shfl_up_sync(0xffffffffu, sp, off);
                if (lane >= off)
                {
                    float nz = oz;
                    int np = op;
                    first_min(nz, np, sz, sp);
                    sz = nz;
                    sp = np;
                }
            }
            float pz = zi; // the running minimum before this lane's chunk
            int pp = i;
            {
                const float ez = __shfl_up_sync(0xffffffffu, sz, 1);
                const int ep = __shfl_up_sync(0xffffffffu, sp, 1);
                if (lane > 0)
                    first_min(pz, pp, ez, ep);
            }
            float tz = zi; // the chain's end over the whole range
            int tpos = i;
            first_min(tz, tpos, __shfl_sync(0xffffffffu, sz, 31), __shfl_sync(0xffffffffu, sp, 31));
            // the samples handed on: the running minimum before the chunk, the
            // chain's end (to position i) and the sample at i
            float hz = zs[pp], hw = ws[pp];
            int hi_ = ids[pp];
            const float end_z = zs[tpos], end_w = ws[tpos];
            const int end_i = ids[tpos];
            const float wi = ws[i];
            const int ii = ids[i];
            __syncwarp();
            if (chain)
            {
                float curz = pz;
                for (int j = lo; j < hi; ++j)
                {
                    const float zj = zs[j];
                    if (zj < curz)
                    {
                        const float wj = ws[j];
                        const int ij = ids[j];
                        zs[j] = hz;
                        ws[j] = hw;
                        ids[j] = hi_;
                        hz = zj;
                        hw = wj;
                        hi_ = ij;
                        curz = zj;
                    }
                }
            }
            const bool moved = chain && tpos != i;
            if (lane == 0)
            {
                if (moved)
                {
                    zs[i] = end_z;
                    ws[i] = end_w;
                    ids[i] = end_i;
                }
                run = __fadd_rn(run, moved ? end_w : wi);
                if (run > center)
                    pick = moved ? end_i : ii;
            }
            pick = __shfl_sync(0xffffffffu, pick, 0);
            __syncwarp();
            if (pick >= 0)
                break;
        }
        if (lane == 0 && pick >= 0)
        {
            const int q = (y0 + pick / ww) * W + x0 + pick % ww;
            plane[3 * (size_t)p] = px[q].x;
            plane[3 * (size_t)p + 1] = px[q].y;
            plane[3 * (size_t)p + 2] = px[q].z;
        }
    }
}

// Weighted median without sorting, for both variants: one block per failed
// pixel. The chosen plane is that of the first sample in (z, window position)
// order whose running weight exceeds half the total. A pivot search finds the
// z value at which the running weight crosses the half (a pivot's side is the
// sum of the weights up to it; samples of one plane share one z at the pixel,
// so there are few distinct values); the weights at that z, in window order
// and in double, then give the sample. What rounding could decide otherwise
// goes to `hard` and through the sorts above:
//   - the samples whose running weight lies within `margin` of the half, if
//     their planes differ. The sort adds up to 1681 doubles (2e-13 of the
//     total), this kernel as many in another order: 1e-11.
//   - GPU_ORDER: that variant's total and running weight are float sums of up
//     to 1681 terms (1681 * 2^-24 = 1.0e-4 of the half each, margin 1.2e-4), and
//     its sort orders equal z values in its own way, so all samples at the
//     crossing z have to share a plane;
//   - a window with a z that is not finite (or the largest float).
// Thread t of the first 123 holds column t % 41 of rows t / 41, + 3, ...: the
// window in row-major order is slot by slot, thread by thread.
// 1440x992 with 376K failed pixels: 3.3 ms, issue bound (58% of the slots; a
// quarter of it the pivot passes), against 43 ms for sorting every window. What
// the GPU order leaves over decides its time: where a window holds a few planes
// (26K pixels at 450x375), nothing or a few pixels, 0.3 - 3.2 ms against 33 - 61; on
// a left-right result of this engine, a plane per superpixel, most pixels: 37 -
// 45 ms against 45 - 54 at 450x375, 102 / 129 at 720x496, 579 / 700 at 1440x992,
// where the CPU order takes 0.5 / 4.1, 1.1 / 10.1 and 5.8 / 52.4. Passes that go
// on until nothing lies between, from a random first pivot, took 3.6 ms. A warp
// per pixel with 53 samples a lane took 6.5 ms (its registers leave no room for
// loads in flight), the pixels' planes and colours read from their own arrays
// (six loads a sample) 5.5, a candidate on either side in every pass 4.2.
constexpr int WS_T = 128, WS_W = WS_T / 32, WS_SIDE = 2 * WM_R + 1, WS_ROWS = WS_T / WS_SIDE;
constexpr int WS_N = (WS_SIDE + WS_ROWS - 1) / WS_ROWS; // samples per thread

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = v + __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Whether the block's marked samples (bit i of a thread's `may`: its slot i)
// all have one plane, and that plane. (x0, y0): the window's corner; every
// thread of the block calls.
__device__ __forceinline__ bool one_plane(const float4 *px, int W, int qx, int qy0, int x0, int y0, unsigned may,
                                          int s_first[WS_W], float4 &pick)
{
    int first = may ? (int)threadIdx.x * 32 + __ffs(may) - 1 : 0x7fffffff;
    first = __reduce_min_sync(0xffffffffu, first);
    if ((threadIdx.x & 31) == 0)
        s_first[threadIdx.x >> 5] = first;
    __syncthreads();
    first = min(min(s_first[0], s_first[1]), min(s_first[2], s_first[3]));
    bool same = first < 0x7fffffff;
    if (same)
    {
        const int t = first >> 5, i = first & 31;
        pick = px[(size_t)(y0 + t / WS_SIDE + WS_ROWS * i) * W + x0 + t % WS_SIDE];
        for (; may; may &= may - 1)
        {
            const float4 v = px[(size_t)(qy0 + WS_ROWS * (__ffs(may) - 1)) * W + qx];
            same = same && __float_as_uint(v.x) == __float_as_uint(pick.x) && __float_as_uint(v.y) == __float_as_uint(pick.y) &&
                   __float_as_uint(v.z) == __float_as_uint(pick.z);
        }
    }
    return __syncthreads_and(same);
}

template <bool GPU_ORDER>
__global__ void __launch_bounds__(WS_T, 8)
    weighted_select_kernel(const float4 *__restrict__ px, const int *__restrict__ list,
                           const int *__restrict__ count, int W, int H, float *__restrict__ plane,
                           const float *__restrict__ wtab, int *__restrict__ hard, int *__restrict__ hard_count)
{
    __shared__ float s_w[766];
    __shared__ float2 s_sum[WS_W];
    __shared__ float s_all[WS_W], s_cand[WS_W];
    __shared__ double s_slot[WS_N][WS_W], s_tot[3][WS_W];
    __shared__ int s_first[WS_W];
    for (int i = threadIdx.x; i < 766; i += WS_T)
        s_w[i] = wtab[i];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nf = *count;
    const int dr = threadIdx.x / WS_SIDE, dc = threadIdx.x % WS_SIDE; // dr == WS_ROWS: no samples
    for (int item = blockIdx.x; item < nf; item += gridDim.x)
    {
        __syncthreads(); // s_w is written; the previous pixel is done with the shared arrays
        const int p = list[item];
        const int y = p / W, x = p - y * W;
        const float colour = px[p].w, fx = (float)x, fy = (float)y;
        const int qx = x - WM_R + dc, qy0 = y - WM_R + dr;
        const bool column = dr < WS_ROWS && qx >= 0 && qx < W;
        float z[WS_N], w[WS_N];
        bool finite = true;
#pragma unroll
        for (int i = 0; i < WS_N; ++i)
        {
            const int qy = qy0 + WS_ROWS * i;
            z[i] = FLT_MAX; // no sample: above every pivot, weight 0
            w[i] = 0.f;
            if (column && qy >= 0 && qy < H && dr + WS_ROWS * i < WS_SIDE)
            {
                const float4 v = px[(size_t)qy * W + qx];
                w[i] = s_w[colour_dist(colour, v.w)];
                z[i] = GPU_ORDER ? __fadd_rn(__fmaf_rn(v.x, fx, __fmul_rn(v.y, fy)), v.z) : get_z(v, fx, fy);
                finite = finite && fabsf(z[i]) < FLT_MAX;
            }
        }
        // weight up to lo <= center < weight up to hi; a pivot whose own weight
        // spans the half ends the search. The first pivot is the pixel's own z
        // (its fill is often the median).
        float total = 0.f;
#pragma unroll
        for (int i = 0; i < WS_N; ++i)
            total = total + w[i];
        total = warp_sum(total);
        if (lane == 0)
            s_all[warp] = total;
        const float4 own = px[p];
        float lo = -FLT_MAX, hi = FLT_MAX;
        float pivot = GPU_ORDER ? __fadd_rn(__fmaf_rn(own.x, fx, __fmul_rn(own.y, fy)), own.z) : get_z(own, fx, fy);
        bool ok = __syncthreads_and(finite);
        const float center = ((s_all[0] + s_all[1]) + (s_all[2] + s_all[3])) * 0.5f;
        for (int pass = 0; ok; ++pass) // block-uniform
        {
            float under = 0.f, upto = 0.f;
#pragma unroll
            for (int i = 0; i < WS_N; ++i)
            {
                if (z[i] < pivot)
                    under = under + w[i];
                if (z[i] <= pivot)
                    upto = upto + w[i];
            }
            under = warp_sum(under);
            upto = warp_sum(upto);
            if (lane == 0)
                s_sum[warp] = make_float2(under, upto);
            __syncthreads();
            under = (s_sum[0].x + s_sum[1].x) + (s_sum[2].x + s_sum[3].x);
            upto = (s_sum[0].y + s_sum[1].y) + (s_sum[2].y + s_sum[3].y);
            if (upto > center)
                hi = pivot;
            else
                lo = pivot;
            if (upto > center && under <= center)
                break;
            // each warp offers a sample strictly between, a lane's in turn; the
            // next pivot is the middle one of the four
            float cand = FLT_MAX;
            unsigned has = 0;
#pragma unroll
            for (int i0 = 0; i0 < WS_N; i0 += 2)
                if (!has)
                {
#pragma unroll
                    for (int i = i0; i < i0 + 2 && i < WS_N; ++i)
                        if (z[i] > lo && z[i] < hi)
                            cand = z[i];
                    has = __ballot_sync(0xffffffffu, cand < FLT_MAX);
                }
            const int r = (5 + 11 * pass) & 31;
            cand = __shfl_sync(0xffffffffu, cand, (__ffs(__funnelshift_r(has, has, r)) - 1 + r) & 31);
            if (lane == 0)
                s_cand[warp] = has ? cand : FLT_MAX;
            __syncthreads();
            // the second of the four in order, the first if it is the only one
            const float a = fminf(s_cand[0], s_cand[1]), b = fmaxf(s_cand[0], s_cand[1]);
            const float c = fminf(s_cand[2], s_cand[3]), d = fmaxf(s_cand[2], s_cand[3]);
            const float second = fminf(fmaxf(a, c), fminf(b, d));
            pivot = second < FLT_MAX ? second : fminf(a, c);
            if (!(pivot < FLT_MAX)) // nothing strictly between: hi is the crossing z
                break;
        }
        if (ok)
        {
            // the total, the weight below hi and the weight at hi in double
            double sums[3] = {0.0, 0.0, 0.0};
            unsigned may = 0; // this thread's samples that may be the one: first all at hi
#pragma unroll
            for (int i = 0; i < WS_N; ++i)
            {
                sums[0] = sums[0] + (double)w[i];
                if (z[i] < hi)
                    sums[1] = sums[1] + (double)w[i];
                if (z[i] == hi)
                {
                    sums[2] = sums[2] + (double)w[i];
                    may |= 1u << i;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                sums[k] = warp_sum(sums[k]);
                if (lane == 0)
                    s_tot[k][warp] = sums[k];
            }
            float4 pick;
            bool same = one_plane(px, W, qx, qy0, x - WM_R, y - WM_R, may, s_first, pick); // synchronises
#pragma unroll
            for (int k = 0; k < 3; ++k)
                sums[k] = (s_tot[k][0] + s_tot[k][1]) + (s_tot[k][2] + s_tot[k][3]);
            const double half = sums[0] * 0.5, eps = (GPU_ORDER ? 1.2e-4 : 1e-11) * sums[0];
            ok = hi < FLT_MAX && sums[1] < half - eps && sums[1] + sums[2] > half + eps;
            if (!GPU_ORDER && ok && !same)
            {
                // several planes at hi: the samples there in window order, and
                // of them those whose running weight meets the half
                double in[WS_N]; // up to this thread within its warp
#pragma unroll
                for (int i = 0; i < WS_N; ++i)
                {
                    double v = z[i] == hi ? (double)w[i] : 0.0;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const double u = __shfl_up_sync(0xffffffffu, v, o);
                        if (lane >= o)
                            v = v + u;
                    }
                    if (lane == 31)
                        s_slot[i][warp] = v;
                    in[i] = v;
                }
                __syncthreads();
                may = 0;
                double run = sums[1];
#pragma unroll
                for (int i = 0; i < WS_N; ++i)
#pragma unroll
                    for (int k = 0; k < WS_W; ++k)
                    {
                        if (k == warp && z[i] == hi && run + in[i] > half - eps && run + in[i] - (double)w[i] <= half + eps)
                            may |= 1u << i;
                        run = run + s_slot[i][k];
                    }
                same = one_plane(px, W, qx, qy0, x - WM_R, y - WM_R, may, s_first, pick);
            }
            ok = ok && same;
            if (ok && threadIdx.x == 0)
            {
                plane[3 * (size_t)p] = pick.x;
                plane[3 * (size_t)p + 1] = pick.y;
                plane[3 * (size_t)p + 2] = pick.z;
            }
        }
        if (!ok && threadIdx.x == 0)
            hard[atomicAdd(hard_count, 1)] = p;
    }
}

__device__ __forceinline__ float median7(float *v)
{
    for (int j = 1; j < 7; ++j)
    {
        float t = v[j];
        int i = j - 1;
        while (i >= 0 && v[i] > t)
        {
            v[i + 1] = v[i];
            i--;
        }
        v[i + 1] = t;
    }
    return v[3];
}

// medianFilter, horizontal pass: interior pixels of D into T (T starts zero).
__global__ void median_h_kernel(const float *D, int W, int H, float *T)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H)
        return;
    int y = i / W, u = i - y * W;
    if (u < 3 || u >= W - 3 || y < 3 || y >= H - 3)
        return;
    if (D[i] >= 0)
    {
        float v[7];
        for (int k = 0; k < 7; ++k)
            v[k] = D[i - 3 + k];
        T[i] = median7(v);
    }
    else
        T[i] = D[i];
}

// vertical pass: reads T (including its untouched zero border rows).
__global__ void median_v_kernel(const float *T, int W, int H, float *D)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H)
        return;
    int y = i / W, u = i - y * W;
    if (u < 3 || u >= W - 3 || y < 3 || y >= H - 3)
        return;
    if (D[i] >= 0)
    {
        float v[7];
        for (int k = 0; k < 7; ++k)
            v[k] = T[(y - 3 + k) * W + u];
        D[i] = median7(v);
    }
}
} // namespace

void launch_lr_check(const float *dispL, const float *dispR, float *planeL, uint8_t *fail,
                     uint8_t *fail2, int W, int H, cudaStream_t st)
{
    int n = W * H;
    lr_fail_kernel<<<ceil_div(n, 256), 256, 0, st>>>(dispL, dispR, W, H, fail);
    note_launch();
    dilate3_kernel<<<ceil_div(n, 256), 256, 0, st>>>(fail, W, H, fail2);
    note_launch();
    lr_fill_kernel<<<ceil_div(n, 256), 256, 0, st>>>(fail, fail2, W, H, planeL);
    note_launch();
    HBP_LAUNCH_CHECK();
}

void launch_plane_to_disp(const float *plane, float *disp, int W, int H, cudaStream_t st)
{
    plane_to_disp_kernel<<<ceil_div(W * H, 256), 256, 0, st>>>(plane, W, H, disp);
    note_launch();
    HBP_LAUNCH_CHECK();
}

// The weighted median of the failed pixels, in place: every kernel reads the
// packed copy. The select kernel, then the variant's sort for what it leaves
// over; both take their lists from the device (a fixed grid walks them), so
// nothing waits for a count.
template <bool GPU_ORDER>
static void weighted_median(const uint8_t *bgr, const uint8_t *fail, float *plane, int W, int H, const float *wtab,
                            Arena &tmp, cudaStream_t st)
{
    const int n = W * H;
    size_t m = tmp.mark();
    float4 *px = tmp.alloc<float4>(n);
    int *list = tmp.alloc<int>(n), *hard = tmp.alloc<int>(n), *counts = tmp.alloc<int>(2);
    HBP_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(int), st));
    pack_and_list<<<ceil_div(n, 256), 256, 0, st>>>(bgr, fail, plane, n, px, list, counts);
    note_launch();
    HBP_LAUNCH_CHECK();
    constexpr int SMS = 148;
    weighted_select_kernel<GPU_ORDER><<<std::min(8 * SMS, n), WS_T, 0, st>>>(px, list, counts, W, H, plane, wtab, hard,
                                                                              counts + 1);
    note_launch();
    if (GPU_ORDER)
        weighted_median_gpu_kernel<<<std::min(5 * SMS, ceil_div(n, WG_W)), 32 * WG_W, 0, st>>>(px, hard, counts + 1, W, H, plane,
                                                                                              wtab);
    else
        weighted_median_kernel<<<std::min(8 * SMS, n), WM_T, 0, st>>>(px, hard, counts + 1, W, H, plane, wtab);
    note_launch();
    HBP_LAUNCH_CHECK();
    tmp.rewind(m);
}

void launch_weighted_median_gpu(const uint8_t *bgr, const uint8_t *fail, float *plane, int W, int H,
                                const float *wtab766, Arena &tmp, cudaStream_t st)
{
    weighted_median<true>(bgr, fail, plane, W, H, wtab766, tmp, st);
}

void median_weight_table(float *host766)
{
    for (int k = 0; k < 766; ++k)
        host766[k] = std::exp(-(float)k / 10.0f);
}

void launch_weighted_median(const uint8_t *bgr, const uint8_t *fail, float *plane, int W, int H, const float *wtab,
                            Arena &tmp, cudaStream_t st)
{
    weighted_median<false>(bgr, fail, plane, W, H, wtab, tmp, st);
}

void launch_driver_median(float *disp, float *tmp, int W, int H, cudaStream_t st)
{
    int n = W * H;
    HBP_CUDA(cudaMemsetAsync(tmp, 0, sizeof(float) * n, st));
    median_h_kernel<<<ceil_div(n, 256), 256, 0, st>>>(disp, W, H, tmp);
    note_launch();
    median_v_kernel<<<ceil_div(n, 256), 256, 0, st>>>(tmp, W, H, disp);
    note_launch();
    HBP_LAUNCH_CHECK();
}

} // namespace hbp
