// Hierarchical min-sum belief propagation over slanted-plane particles on the
// image segmentation pyramid. Reference: HBP_ISP (hbp_isp.hpp:122-442,
// hbp_isp.cu:1-1346).
//
// Per node K = 12 plane slots: 0-3 best, 4-7 prior (the parent's best), 8-11
// candidates. Coarse to fine, each level runs (10 + 10*level) outer
// iterations of {4 x RANSAC, 1 x spatial propagation, [1 x random adjust]}
// candidate steps; after each, the candidates' data cost is computed and one
// BP sweep passes, smooths, normalises and aggregates messages, then keeps
// the P best slots per node.
//
// Engine layout (node-major / edge-major, so the neighbour gathers of the BP
// kernels read contiguous slots): plane[n][12] float4, cost/belief[n][12],
// msg/msg_t[e][12]. Each level lists its pixels sorted by node, raster order
// inside a node (packed y<<16|x); the data cost walks that list in windows of
// 256 positions, and a node's chunks are the windows it overlaps.
//
// Reduction orders (the reference's float atomics / reduce_by_key have none):
// plane costs by the segmented-scan order described at k_cost; beliefs =
// cost + out-edge messages in edge order.
// Everything else follows the reference operation for operation; this file is
// compiled without multiply-add contraction, so each a*b+c rounds twice like
// the CPU oracle except where a fused multiply-add is written out
// (__fmaf_rn: the data cost's plane evaluation and interpolation, the
// smoothness term and the message sum).
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <memory>
#include <vector>

#include <cuda_fp16.h>

#include "engine.h"

namespace hbp
{
namespace
{
struct LevelDev
{
    int N, E, Nh, nchunks;
    const int *clus;         // N -> parent
    const uint32_t *pix;     // HW packed y<<16|x, sorted by (node, pixel)
    const int *pix_off;      // N + 1
    const int *chunk_off;    // N + 1: first data-cost chunk of each node
    const int *pnode;        // HW: node of each list position
    const int2 *win;         // per 256-position window: its first node (~node: fills it) and chunk
    const int2 *bd;          // E
    const int *bdl;          // E
    const int *nb_off;       // N + 1
    const int *rev;          // E
    const float *dc;         // 2E: colour weight, centroid distance
    const float *mx, *my;    // N: centroid
    const uint32_t *child;   // N: this level's nodes grouped by parent
    const int *child_off;    // Nh + 1
    float4 *plane;           // N x K
    float *cost, *belief;    // N x K
    int4 *pid;               // N: RANSAC points (packed y<<16|x)
    unsigned long long *keep; // N: kept slots (count | 4-bit indices)
};

struct Common
{
    int W, H, D, TX; // TX: volume tiles per row
    float lambda, tau, tau_smooth; // tau: the data cost outside [0, D-1)
    const uint8_t *vol; // tiled, vol_offset() (Census: uint8 costs)
    const float *volf;  // or the same layout in floats (MC-CNN); null for uint8
    const float *wta;   // HW
};

// The BP kernels of a stream follow one another at once, so each is launched
// with programmatic stream serialization: it may start while its predecessor
// still runs, reads what the level's setup wrote (pixel lists, edges, offsets)
// and waits here for the predecessor to finish before it touches planes,
// costs, beliefs or messages. Every kernel of the chain waits in every thread
// that reads or writes such data, so a finished kernel implies finished
// predecessors. When this came in, the BP of a 720x496 pair went from 48.6 to
// 35.0 ms, of a 96x64 pair from 22.4 to 14.6.
__device__ __forceinline__ void after_predecessor()
{
    cudaGridDependencySynchronize();
}
__device__ __forceinline__ void let_successor_start()
{
    cudaTriggerProgrammaticLaunchCompletion();
}
template <typename Desc>
void launch_chained(void (*kernel)(Desc), int grid, int block, cudaStream_t st, const Desc &d, size_t smem = 0)
{
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.stream = st;
    c.dynamicSmemBytes = smem;
    c.attrs = &a;
    c.numAttrs = 1;
    HBP_CUDA(cudaLaunchKernelEx(&c, kernel, d));
    note_launch();
}

__device__ __forceinline__ int px_x(uint32_t xy) { return (int)(xy & 0xffffu); }
__device__ __forceinline__ int px_y(uint32_t xy) { return (int)(xy >> 16); }

// A byte as float without the conversion pipe: the bits 0x4B000000 | v are
// the float 2^23 + v, so subtracting 2^23 gives v exactly.
__device__ __forceinline__ float byte_to_float(uint32_t v)
{
    return __uint_as_float(0x4B000000u | v) - 8388608.0f;
}

// What the data cost of one view and level reads: a launch carries it in its
// parameters, so that a block's first loads are the pixel list itself.
struct CostArgs
{
    const uint32_t *pix; // the level's pixel list
    const int *pnode;
    const int2 *win;     // per window: first node (whole windows: ~node), its chunk
    const float4 *plane; // the planes' node records (K per node), at the first slot read
    const int *clus;     // COST_INIT: the planes are the parents', else null
    float4 *pc;          // chunk sums
    const uint8_t *vol;  // tiled, vol_offset() (Census: uint8 costs)
    const float *volf;   // or the same layout in floats (MC-CNN); null for uint8
    int HW, N, TX, D;
    float lambda, tau;
};

// read_plane_cost (hbp_isp.cu:205-227) of one plane at one pixel, in two
// halves: the two volume reads are issued by fetch() and used by cost(), so
// that a lane can have many in flight. They are predicated by hand: as an `if`
// some of them became branches, and the reads behind a branch wait for those
// before it (data cost of sixteen 720x496 views 144 -> 139 ms, BP of a
// 1440x992 view 84.6 -> 80.3). For d in [0, D-1), (float)(d + 1) == (float)d +
// 1 exactly.
// F32: the float volume of the MC-CNN / AD paths (volf), else the uint8
// Census volume (vol); a template parameter, so the Census path carries no
// branch on the volume's type.
struct PixelAt
{
    float xf, yf;
    size_t base; // vol_tile_base

    __device__ __forceinline__ PixelAt(const CostArgs &c, uint32_t xy)
    {
        const int x = px_x(xy), y = px_y(xy);
        xf = (float)x;
        yf = (float)y;
        base = vol_tile_base(x, y, c.TX, c.D);
    }
};
template <bool F32>
struct PlaneCost
{
    float d_f;
    uint32_t v0, v1; // a volume value's bits: a byte, or a float

    // v0 and v1 from rows d (at address pv) and d + 1 of a tile, or 0. An
    // integer: outside the volume it is never read.
    __device__ __forceinline__ void read_if(bool in, uint64_t pv)
    {
        if constexpr (F32)
            asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t"
                "@q ld.global.nc.u32 %0, [%2];\n\t@q ld.global.nc.u32 %1, [%2 + %4];\n\t}"
                : "=&r"(v0), "=&r"(v1)
                : "l"(pv), "r"((unsigned)in), "n"(VT_BYTES * sizeof(float)));
        else
            asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t"
                "@q ld.global.nc.u8 %0, [%2];\n\t@q ld.global.nc.u8 %1, [%2 + %4];\n\t}"
                : "=&r"(v0), "=&r"(v1)
                : "l"(pv), "r"((unsigned)in), "n"(VT_BYTES));
    }

    __device__ __forceinline__ void fetch(const CostArgs &c, const PixelAt &px, float4 pl)
    {
        d_f = __fmaf_rn(pl.x, px.xf, __fmaf_rn(pl.y, px.yf, pl.z));
        const int d = __float2int_rd(d_f);
        const bool in = (unsigned)d < (unsigned)(c.D - 1);
        const uint64_t row = px.base + vol_row_offset(d);
        if constexpr (F32)
            read_if(in, reinterpret_cast<uint64_t>(c.volf) + row * sizeof(float));
        else
            read_if(in, reinterpret_cast<uint64_t>(c.vol) + row);
    }
    __device__ __forceinline__ float cost(const CostArgs &c) const
    {
        const int d = __float2int_rd(d_f);
        const float a = F32 ? __uint_as_float(v0) : byte_to_float(v0);
        const float b = F32 ? __uint_as_float(v1) : byte_to_float(v1);
        const float fd = (float)d;
        const float in = __fmaf_rn((fd + 1.0f) - d_f, a, (d_f - fd) * b);
        return c.lambda * ((unsigned)d < (unsigned)(c.D - 1) ? in : c.tau);
    }
};

// ---------------------------------------------------------------------------
// level setup
__global__ void iota_xy(uint32_t *key, uint32_t *val, const int *im_clus, int W, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        key[i] = (uint32_t)im_clus[i];
        val[i] = ((uint32_t)(i / W) << 16) | (uint32_t)(i % W);
    }
}

__global__ void compose_im_clus(const int *im, const int *clus, int n, int *out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = clus[im[i]];
}

__global__ void iota_int(int *v, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        v[i] = i;
}

// First list position of every node from the sorted node keys (every node
// holds at least one pixel): off[key[i]] = i where a run of equal keys
// starts, off[N] = n. No atomics: at coarse levels a count by atomics put
// every pixel on a handful of counters.
__global__ void run_starts(const uint32_t *key, int n, int N, int *off)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && (i == 0 || key[i] != key[i - 1]))
        off[key[i]] = i;
    if (i == 0)
        off[N] = n;
}

// A node's data-cost chunks are the 256-position windows of the level's pixel
// list that it overlaps.
__global__ void chunk_counts(const int *pix_off, int N, int *nch)
{
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < N)
        nch[n] = ((pix_off[n + 1] - 1) / PC_CHUNK) - (pix_off[n] / PC_CHUNK) + 1;
    if (n == N)
        nch[N] = 0;
}

// Per window of the pixel list its first node n (complemented if the node
// fills the window) and n's chunk there. The windows' nodes are consecutive
// (the list is sorted and no node is empty), and so are their chunks.
__global__ void window_info(const uint32_t *key, const int *pix_off, const int *chunk_off, int n, int2 *win)
{
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    const long q0 = (long)w * PC_CHUNK;
    if (q0 >= n)
        return;
    const int k = (int)key[q0];
    const bool whole = q0 + PC_CHUNK <= n && (int)key[q0 + PC_CHUNK - 1] == k;
    win[w] = make_int2(whole ? ~k : k, chunk_off[k] + w - pix_off[k] / PC_CHUNK);
}

// reverse_bd_id_k (hbp_isp.cu:154-175): first edge t -> s in t's range.
__global__ void reverse_ids(const int2 *bd, const int *nb_off, int E, int *rev)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E)
        return;
    int2 st = bd[e];
    int r = 0;
    for (int k = nb_off[st.y]; k < nb_off[st.y + 1]; ++k)
        if (bd[k].y == st.x)
        {
            r = k;
            break;
        }
    rev[e] = r;
}

// sum_to_mean + compute_dist_color_pos + dist_trans (hbp_isp.cu:78-126,
// :952-970): colour weight exp(-(|dL| + |da| + |db|) / 20), computed in double
// and rounded once; centroid distance sqrt(dx^2 + dy^2).
__global__ void level_means(const float *sums, int N, float *mx, float *my, float *ml)
{
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N)
        return;
    float w = sums[5 * (size_t)N + n];
    for (int c = 0; c < 3; ++c)
        ml[(size_t)c * N + n] = sums[(size_t)c * N + n] / w;
    mx[n] = sums[3 * (size_t)N + n] / w;
    my[n] = sums[4 * (size_t)N + n] / w;
}

__global__ void edge_weights(const int2 *bd, int E, int N, const float *ml, const float *mx,
                             const float *my, float *dc)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E)
        return;
    int s = bd[e].x, t = bd[e].y;
    float col = fabsf(ml[s] - ml[t]) + fabsf(ml[N + s] - ml[N + t]);
    col = col + fabsf(ml[2 * (size_t)N + s] - ml[2 * (size_t)N + t]);
    float dx = mx[s] - mx[t], dy = my[s] - my[t];
    float pos = dx * dx + dy * dy;
    dc[e] = (float)exp((double)(-col / 20.0f));
    dc[E + e] = sqrtf(pos);
}

// ---------------------------------------------------------------------------
// candidates
__device__ __forceinline__ float4 fit_plane(float Ax, float Ay, float Az, float Bx, float By, float Bz,
                                            float Cx, float Cy, float Cz)
{
    // fit_plane_from_points (hbp_isp.cu:531-548)
    float ax = Bx - Ax, ay = By - Ay, az = Bz - Az;
    float bx = Cx - Ax, by = Cy - Ay, bz = Cz - Az;
    float nx = ay * bz - az * by;
    float ny = az * bx - ax * bz;
    float nz = ax * by - ay * bx;
    nx /= nz;
    ny /= nz;
    nz /= nz;
    if (fabsf(nz - 1.f) > FLT_EPSILON)
        return make_float4(0.f, 0.f, (Az + Bz + Cz) / 3.f, 0.f);
    return make_float4(-nx, -ny, nx * Ax + ny * Ay + Az, 0.f);
}



// ---------------------------------------------------------------------------
// Batched BP. A batch holds up to MAXV views (one view = one pyramid + cost
// volume; a pair contributes one, or two with the right view). Every kernel
// below serves one BP phase of every participating view at once: items
// (nodes, chunks, edges) of the views are laid end to end and each thread or
// warp finds its view from the prefix table of the launch's step descriptor.
//
// A BP step of the reference (generate_plane, compute_plane_cost,
// belief_propagation; hbp_isp.cu:1206-1311) runs as
//   node phase   select of the previous step (aggregate_belief_k,
//                get_belief_order, select_belief) fused with the step's RANSAC
//                or random-adjust candidates, four lanes or a block per node;
//   [spatial]    select_child, neighbor, set_candidate, one thread per node and
//                candidate;
//   then the next two, in one launch while few windows are in flight:
//   data cost    read_plane_cost + the per-node reduction, a block per
//                256-position window;
//   edge phase   passing_msg + smooth_msg + normalize_msg, one thread, four or
//                eight lanes per edge, with the previous step's messages pulled through
//                ping_pang_msg + select_msg (msg[e] = msg_t[rev e] compacted by
//                the kept slots of e's target).
struct ViewBufs
{
    void *msgt[2]; // [E][K] ping-pong: float, or __half when fp16
    int fp16;      // messages stored as FP16 (FP32 arithmetic)
    float4 *pc[2];  // chunk partial costs ping-pong
};

struct ViewDev
{
    Common c;
    const LevelDev *lv; // [L]
    ViewBufs b;
    float *disp, *plane_out;
    float *lvl_disp, *lvl_plane; // per-level maps (run_ms_vis), index L-1-li; null if not kept
    int L;
};

constexpr int MAXV = 16; // tasks per launch descriptor

enum NodeMode
{
    NODE_SELECT = 0,
    NODE_SELECT_RANSAC = 1,
    NODE_SELECT_RANDOM = 2
};

struct Task
{
    const ViewDev *vd;             // the view's record in device memory
    const LevelDev *lvl, *lvh;     // its level li and li+1 records
    int v, li;
    int first;        // first BP step of the level: no select, zero messages
    int pb, mb;       // cost partials written / messages written
    int mode;         // node phase: NodeMode
};

struct StepDesc
{
    int nt;
    int pre[MAXV + 1];
    Task t[MAXV];
};

__device__ __forceinline__ int find_task(const StepDesc &d, int item)
{
    int k = 0;
    while (k + 1 < d.nt && item >= d.pre[k + 1])
        ++k;
    return k;
}

// S3 of the data-cost order: a node's chunk sums c0..c1-1 added in order;
// the loads are issued 8 at a time (the additions stay sequential).
__device__ __forceinline__ float4 sum_chunks(const float4 *pc, int c0, int c1)
{
    float4 a = pc[c0];
    int ch = c0 + 1;
    for (; ch + 8 <= c1; ch += 8)
    {
        float4 q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            q[j] = pc[ch + j];
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            a.x = a.x + q[j].x;
            a.y = a.y + q[j].y;
            a.z = a.z + q[j].z;
            a.w = a.w + q[j].w;
        }
    }
    for (; ch < c1; ++ch)
    {
        const float4 q = pc[ch];
        a.x = a.x + q.x;
        a.y = a.y + q.y;
        a.z = a.z + q.z;
        a.w = a.w + q.w;
    }
    return a;
}

// ---------------------------------------------------------------------------
// Node phase: select of the previous step (aggregate_belief_k,
// get_belief_order, select_belief; hbp_isp.cu:405-417, :432-472), then the
// step's RANSAC or random-adjust candidates.
//
// Four lanes per node: lane j < 3 owns slots 4j .. 4j+3 (a slot's belief is a
// serial sum: cost, then the out-edge messages in edge order; S3 of the data
// cost for the candidate slots), lane p draws candidate p. Levels of large
// nodes (8 chunks and more on average) take a block per node: its threads
// bring the chunk sums and messages into shared memory, so that the serial
// sums run from there.
// Per launch of sixteen 720x496 views at levels 2 / 3 / 5 / 6 / 7 (with the
// events' 5 us): 48 / 20 / 15 / 12 / 15 us. A thread per node (a warp per node
// of 16 chunks and more), 12 sums, 24 scattered reads and 66 comparisons in
// one chain, took 51 / 22 / 25 / 17 / 25; sixteen lanes per node, one per
// slot, 106 / 32 / 15 / 11 / 12: the ranks, the draws and the plane fit then
// issue for two nodes per warp instead of eight.
struct NodeArgs
{
    const int *nb_off, *chunk_off, *pix_off;
    const float4 *pc;    // the previous step's chunk sums
    const void *msg;     // the previous step's messages [E][K], float or __half
    float4 *plane;       // N x K
    float *cost, *belief; // N x K (cost: slots 0-7 live here; belief: 0-7)
    int4 *pid;
    unsigned long long *keep;
    const uint32_t *pix;
    const float *wta;
    const float *mx, *my;
    int N, W, fp16, first, mode, block_per_node;
    // the generator's state: after the level's earlier draws a node's generator
    // holds seed_a * pix_off[n] + seed_c (mod 2^31)
    uint32_t seed_a, seed_c;
    float max_dz, max_dn;
};
struct NodeDesc
{
    int nt;
    int pre[MAXV + 1]; // blocks before each task
    NodeArgs t[MAXV];
};
constexpr int NODE_T = 128, NODE_LANES = 4, NODE_PER_BLOCK = NODE_T / NODE_LANES;
constexpr int NODE_BLOCK_CHUNKS = 8; // chunks per node from which a level's nodes take a block each (4: 48 ms per batch, 8: 44)
constexpr int NODE_BLOCK_NODES = 1200; // nodes per launch up to which each takes a block anyway: the chip has room, and a
                                       // block's reads are all in flight at once (720x496 pair 24.8 -> 23.5 ms of BP)
constexpr int NODE_TILE = NODE_T; // chunk sums staged at a time, one per thread
constexpr int NODE_MSGS = 32;     // messages staged
constexpr size_t NODE_SMEM = sizeof(float4) * (NODE_TILE + NODE_MSGS * (K / 4)); // of a launch with nodes that take a block

// k steps of the generator at once: s -> a * s + c (mod 2^31)
struct LcgJump
{
    uint32_t a = 1, c = 0;
    __host__ __device__ constexpr LcgJump(int k)
    {
        for (int i = 0; i < k; ++i)
        {
            a = 1103515245u * a;
            c = 1103515245u * c + 12345u;
        }
    }
    __host__ __device__ __forceinline__ uint32_t operator()(uint32_t s) const { return (a * s + c) & 0x7fffffffu; }
    void then(LcgJump j) // this jump, then j
    {
        a = j.a * a;
        c = j.a * c + j.c;
    }
};
// the generator's state after 0, K, 2K or 3K draws
template <int DRAWS>
__device__ __forceinline__ uint32_t lcg_ahead(uint32_t s, int p)
{
    constexpr LcgJump j1(DRAWS), j2(2 * DRAWS), j3(3 * DRAWS);
    return p == 0 ? s : p == 1 ? j1(s) : p == 2 ? j2(s) : j3(s);
}

// slots 4j .. 4j+3 of message e as floats
__device__ __forceinline__ float4 msg4_at(const NodeArgs &t, size_t e, int j)
{
    if (!t.fp16)
        return static_cast<const float4 *>(t.msg)[e * (K / 4) + j];
    const uint2 w = static_cast<const uint2 *>(t.msg)[e * (K / 4) + j];
    const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&w.x));
    const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&w.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}

__device__ __forceinline__ float4 add4(float4 a, float4 b)
{
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// Candidate p's plane and its three points (ransac_candidate_plane +
// make_three_diff_id + fit_plane_from_points, hbp_isp.cu:504-548, :592-640).
__device__ __forceinline__ float4 ransac_plane(const NodeArgs &t, int n, int p, uint32_t xy[3])
{
    const int cp = t.pix_off[n], cn = t.pix_off[n + 1] - cp;
    uint32_t s = lcg_ahead<3>((t.seed_a * (uint32_t)cp + t.seed_c) & 0x7fffffffu, p);
    s = lcg(s);
    const int p0 = (int)(s % (uint32_t)cn);
    s = lcg(s);
    int p1 = cn > 1 ? (int)(s % (uint32_t)(cn - 1)) : 0;
    s = lcg(s);
    int p2 = cn > 2 ? (int)(s % (uint32_t)(cn - 2)) : 0;
    if (cn <= 3)
    {
        p1 = (p0 + 1) % cn;
        p2 = (p1 + 1) % cn;
    }
    else
    {
        if (p1 == p0)
            p1 = cn - 1;
        if (p2 == p0)
            p2 = (p1 == cn - 2) ? cn - 1 : cn - 2;
        else if (p2 == p1)
            p2 = (p0 == cn - 2) ? cn - 1 : cn - 2;
    }
    xy[0] = t.pix[cp + p0];
    xy[1] = t.pix[cp + p1];
    xy[2] = t.pix[cp + p2];
    float z[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        z[j] = t.wta[(size_t)px_y(xy[j]) * t.W + px_x(xy[j])];
    return fit_plane((float)px_x(xy[0]), (float)px_y(xy[0]), z[0], (float)px_x(xy[1]), (float)px_y(xy[1]), z[1],
                     (float)px_x(xy[2]), (float)px_y(xy[2]), z[2]);
}

// random_candidate_plane + normalize_plane (hbp_isp.cu:495-503, :641-674) for
// candidate p of node n
__device__ __forceinline__ float4 random_plane(const NodeArgs &t, int n, int p, float4 pl)
{
    const float x = t.mx[n], y = t.my[n];
    uint32_t s = lcg_ahead<4>((t.seed_a * (uint32_t)t.pix_off[n] + t.seed_c) & 0x7fffffffu, p);
    float z = pl.x * x + pl.y * y + pl.z;
    s = lcg(s);
    float dz = (float)s / 2147483648.0f * t.max_dz;
    z += dz;
    s = lcg(s);
    float dnx = (float)s / 2147483648.0f * t.max_dn;
    s = lcg(s);
    float dny = (float)s / 2147483648.0f * t.max_dn;
    s = lcg(s);
    float dnz = (float)s / 2147483648.0f * t.max_dn;
    float norm = sqrtf(pl.x * pl.x + pl.y * pl.y + pl.z * pl.z);
    pl.x /= norm;
    pl.y /= norm;
    pl.z /= norm;
    pl.x += dnx;
    pl.y += dny;
    pl.z += dnz;
    float a = -pl.x / pl.z, b = -pl.y / pl.z;
    float cc = z - a * x - b * y;
    return make_float4(a, b, cc, 0.f);
}

// The rest of a node's phase by its four lanes (mask gm), lane j < 3 holding
// the costs cs and beliefs b of its slots: rank (a later slot loses ties),
// move the kept slots to the front in slot order, record which, then candidate
// j (drawn from the points xy).
__device__ __forceinline__ void node_finish(const NodeArgs &t, int n, int j, unsigned gm, float4 cs4, float4 b4,
                                            const uint32_t xy[3], float4 drawn)
{
    float4 *pl = t.plane + (size_t)n * K;
    if (!t.first)
    {
        const float cs[4] = {cs4.x, cs4.y, cs4.z, cs4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
        int ord[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < K; ++q)
        {
            const float bq = __shfl_sync(gm, b[q & 3], q >> 2, NODE_LANES);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                ord[i] += q < 4 * j + i ? !(b[i] < bq) : (bq < b[i]); // q == 4j + i: bq < b[i] is false
        }
        unsigned m = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            m |= (unsigned)(j < K / 4 && ord[i] < P) << (4 * j + i);
        m |= __shfl_xor_sync(gm, m, 1);
        m |= __shfl_xor_sync(gm, m, 2);
        const int nb = __popc(m);
        float4 v[4];
        int to[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const int k = 4 * j + i;
            to[i] = (m >> k) & 1u ? __popc(m & ((1u << k) - 1u)) : NODE_LANES * 4; // not kept: above every k
            if (to[i] < k)
                v[i] = pl[k];
        }
        __syncwarp(gm); // every slot that moves is read before one is written
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const int k = 4 * j + i;
            if (to[i] < k)
                pl[to[i]] = v[i];
            // slots the kept ones do not fill keep their cost, and their
            // belief is their own; consumers read slots 0-7
            if (to[i] < k && to[i] < 2 * P)
                t.cost[(size_t)n * K + to[i]] = cs[i];
            if (to[i] < 2 * P)
                t.belief[(size_t)n * K + to[i]] = b[i];
            if (k >= nb && k < 2 * P)
                t.belief[(size_t)n * K + k] = b[i];
        }
        if (j == 3)
        {
            unsigned long long kl = (unsigned long long)nb;
            int i = 0;
            for (unsigned r = m; r; r &= r - 1)
                kl |= (unsigned long long)(__ffs(r) - 1) << (4 + 4 * i++);
            t.keep[n] = kl;
        }
        __syncwarp(gm);
    }
    if (t.mode == NODE_SELECT_RANSAC)
    {
        pl[2 * P + j] = drawn;
        if (j == P - 1)
            t.pid[n] = make_int4((int)xy[0], (int)xy[1], (int)xy[2], 0);
    }
    else if (t.mode == NODE_SELECT_RANDOM)
        pl[2 * P + j] = random_plane(t, n, j, pl[2 * P + j]);
}

__device__ __forceinline__ void node_lanes(const NodeArgs &t, int n, int j)
{
    if (n >= t.N) // uniform over the node's lanes
        return;
    const unsigned gm = 0xfu << (threadIdx.x & 28);
    uint32_t xy[3];
    float4 cs = make_float4(0.f, 0.f, 0.f, 0.f), b = cs, drawn = cs;
    if (t.mode == NODE_SELECT_RANSAC)
        drawn = ransac_plane(t, n, j, xy);
    const int c0 = t.chunk_off[n], c1 = t.chunk_off[n + 1], e1 = t.nb_off[n + 1];
    int e = t.nb_off[n];
    after_predecessor();
    if (!t.first && j < K / 4)
    {
        if (j < 2)
            cs = reinterpret_cast<const float4 *>(t.cost)[(size_t)n * (K / 4) + j];
        else
            cs = sum_chunks(t.pc, c0, c1);
        b = cs;
        for (; e + 4 <= e1; e += 4) // reads 4 at a time
        {
            float4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                v[i] = msg4_at(t, (size_t)(e + i), j);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                b = add4(b, v[i]);
        }
        for (; e < e1; ++e)
            b = add4(b, msg4_at(t, (size_t)e, j));
    }
    node_finish(t, n, j, gm, cs, b, xy, drawn);
}

__device__ __forceinline__ void node_block(const NodeArgs &t, int n, float4 *s_pc, float4 *s_msg)
{
    const int j = threadIdx.x;
    uint32_t xy[3];
    float4 cs = make_float4(0.f, 0.f, 0.f, 0.f), b = cs, drawn = cs;
    if (t.mode == NODE_SELECT_RANSAC && j < NODE_LANES)
        drawn = ransac_plane(t, n, j, xy);
    const int e0 = t.nb_off[n], e1 = t.nb_off[n + 1], em = min(e1, e0 + NODE_MSGS);
    const int c0 = t.chunk_off[n], c1 = t.chunk_off[n + 1];
    after_predecessor();
    if (!t.first) // block-uniform
    {
        if (j < 2)
            cs = reinterpret_cast<const float4 *>(t.cost)[(size_t)n * (K / 4) + j];
        float4 nx;
        if (c0 + j < c1)
            nx = t.pc[c0 + j];
        for (int i = j; i < (em - e0) * (K / 4); i += NODE_T)
            s_msg[i] = msg4_at(t, (size_t)e0 + i / (K / 4), i % (K / 4));
        for (int c = c0; c < c1; c += NODE_TILE)
        {
            __syncthreads(); // the previous tile is summed
            s_pc[j] = nx;
            __syncthreads();
            if (c + NODE_TILE + j < c1)
                nx = t.pc[c + NODE_TILE + j];
            if (j == 2) // S3: the chunk sums in chunk order
            {
                const int cnt = min(NODE_TILE, c1 - c);
                int i = c == c0;
                if (i)
                    cs = s_pc[0];
#pragma unroll 8
                for (; i < cnt; ++i)
                    cs = add4(cs, s_pc[i]);
            }
        }
        if (j < K / 4)
        {
            b = cs;
#pragma unroll 8
            for (int e = 0; e < em - e0; ++e)
                b = add4(b, s_msg[e * (K / 4) + j]);
            for (int e = em; e < e1; ++e)
                b = add4(b, msg4_at(t, (size_t)e, j));
        }
    }
    if (j < NODE_LANES)
        node_finish(t, n, j, 0xfu, cs, b, xy, drawn);
}

__global__ void __launch_bounds__(NODE_T) k_node(const __grid_constant__ NodeDesc d)
{
    extern __shared__ float4 s_node[]; // NODE_SMEM, if a task has nodes that take a block
    let_successor_start();
    int ti = 0;
    while (ti + 1 < d.nt && (int)blockIdx.x >= d.pre[ti + 1])
        ++ti;
    const NodeArgs &t = d.t[ti];
    const int blk = blockIdx.x - d.pre[ti];
    if (t.block_per_node) // uniform per task
        node_block(t, blk, s_node, s_node + NODE_TILE);
    else
        node_lanes(t, blk * NODE_PER_BLOCK + threadIdx.x / NODE_LANES, threadIdx.x % NODE_LANES);
}

// Spatial candidates (select_child_plane, neighbor_candidate_plane and
// set_candidate_plane_k, hbp_isp.cu:676-741): candidate p of every child of
// parent id is the best plane of a random child of a random neighbour of id.
// The reference draws each parent's random child first, then each parent's
// random neighbour, then hands the result to the children; the draws follow
// from the parents' numbers and the draws before, so a thread per (node,
// candidate) draws both for itself and the three launches are one.
struct SpatialArgs
{
    const int *clus;                   // node -> parent
    const int *nb_off;                 // this level's: seeds the neighbour draws, by parent number
    const int *h_nb_off;               // the parents' edges
    const int2 *h_bd;
    const uint32_t *child;
    const int *child_off;
    float4 *plane; // N x K
    int N;
    uint32_t seed_a, seed_c; // a generator's state: seed_a * s0 + seed_c (mod 2^31), s0 = nb_off[id] or child_off[id]
};
struct SpatialDesc
{
    int nt;
    int pre[MAXV + 1]; // blocks before each task
    SpatialArgs t[MAXV];
};
constexpr int SPATIAL_T = 128;
__global__ void __launch_bounds__(SPATIAL_T) k_spatial(const __grid_constant__ SpatialDesc d)
{
    let_successor_start();
    int ti = 0;
    while (ti + 1 < d.nt && (int)blockIdx.x >= d.pre[ti + 1])
        ++ti;
    const SpatialArgs &t = d.t[ti];
    const int i = (blockIdx.x - d.pre[ti]) * SPATIAL_T + threadIdx.x, n = i / P, p = i % P;
    if (n >= t.N)
        return;
    auto draw = [&](int s0) { return lcg(lcg_ahead<1>((t.seed_a * (uint32_t)s0 + t.seed_c) & 0x7fffffffu, p)); };
    int id = t.clus[n];
    const int nbp = t.h_nb_off[id], nbn = t.h_nb_off[id + 1] - nbp;
    if (nbn > 0)
        id = t.h_bd[nbp + (int)(draw(t.nb_off[id]) % (uint32_t)nbn)].y;
    const int cp = t.child_off[id], cn = t.child_off[id + 1] - cp;
    const int ch = (int)t.child[cp + (int)(draw(cp) % (uint32_t)cn)];
    after_predecessor();
    t.plane[(size_t)n * K + 2 * P + p] = t.plane[(size_t)ch * K];
}

// COST_INIT: priors of the parent's best slots (init_bp, hbp_isp.cu:930-950);
// COST_STEP: candidates in slots 8-11.
enum CostMode
{
    COST_INIT = 0,
    COST_STEP = 1
};

// Data cost of 4 planes (read_plane_cost for every pixel, hbp_isp.cu:205-227,
// and the per-node sum of compute_plane_cost, :1159-1174). One block = one
// 256-position window of the level's pixel list (sorted by node, raster order
// inside a node). The node sum is taken in a fixed order (the reference's float atomics have none; the CPU oracle
// restates it):
//   S0 a window that one node fills: slot j sums positions j, j+32, ...,
//      j+224 in order, then an xor butterfly (offsets 16..1) over the slots;
// any other window is cut into 8 sub-windows of 32 positions:
//   S1 inside each 32-position sub-window the pixels of one node form a
//      segment, summed by a segmented Hillis-Steele scan: for off = 1, 2, 4,
//      8, 16, x[r] = x[r - off] + x[r] where r - off is still in the segment;
//   S2 inside the 256-window the node's S1 pieces are added in order (a
//      sub-window whose first segment continues its predecessors' last one
//      adds their pieces, kept in shared memory, before its own);
//   S3 the node's 256-window sums (its chunks, pc[]) are added in chunk order
//      by the consumers (k_init_nodes, k_node).
constexpr int SUBS = PC_CHUNK / 32; // sub-windows of a window
// A block of four warps takes a window. A whole one: a warp per plane, which
// keeps its sums to itself (no shared memory, no barrier); a mixed one: two
// sub-windows per warp with all four planes (the segments are found once).
// 12 blocks per SM (40 registers): the volume's scattered bytes come from L2
// and HBM, so the kernel lives on the number of reads in flight, 48 warps of 8
// or 16 reads a lane. What limits it then: single 32-byte sectors from HBM (4.0
// - 4.1 TB/s, 0.61 - 0.63 of a copy's rate, in the captures of eight views at
// levels 2 and 5; L2 hits 26%), with a ramp and a tail of a fifth of the launch.
// Issue (53 - 57%) and the L1's data pipe (52 - 64%, 5 wavefronts a gather) have room.
// Per launch of sixteen 720x496 D128 views at levels 2 / 5 / 7, and data cost
// per batch: 76 / 62 / 56 us, 139 ms. A warp per window (a serial walk of 8
// sub-windows, 64 registers, 32 warps) took 94 / 75 / 63, 166 ms. Before the
// reads were predicated by hand, this form took 76 / 66 / 60, 145; whole
// windows split by positions too, meeting in shared memory, 80 / 68 / 60, 149;
// 16 reads a lane for whole windows 82 / 74 / 66, 158; two warps a window 101
// / 74 / 62, 172; several windows per block 171 - 196 ms. The conversions of
// the pixel and of the floor on the FP32 and ALU pipes instead of the
// conversion pipe: 152 ms (a quarter of that pipe is in use, half of the ALU).
constexpr int COST_SUBS = 2;
constexpr int COST_T = PC_CHUNK / COST_SUBS, COST_MIN_BLOCKS = 12;

struct CostShared // of a mixed window's sub-windows
{
    float4 tail[SUBS]; // S1 sum of the last segment
    int first[SUBS], last[SUBS], whole[SUBS]; // first and last node, whether one fills it
};
static_assert(COST_T / 32 == P, "a warp per plane");

// DEPTH: positions of a whole window whose reads a lane has in flight
template <bool F32, int DEPTH>
__device__ __forceinline__ void cost_window(const CostArgs &c, int win, CostShared &sh)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 wi = c.win[win];
    if (wi.x < 0) // block-uniform: one node fills the window
    {
        // warp w: plane w at every position, lane j the slots' sums
        const uint32_t *pix = c.pix + win * PC_CHUNK + lane;
        uint32_t xy[SUBS];
#pragma unroll
        for (int k = 0; k < SUBS; ++k)
            xy[k] = pix[32 * k];
        const float4 *src = c.plane + (size_t)(c.clus ? c.clus[~wi.x] : ~wi.x) * K + w;
        after_predecessor();
        const float4 pl = *src;
        float a = 0.f;
#pragma unroll
        for (int k0 = 0; k0 < SUBS; k0 += DEPTH)
        {
            PlaneCost<F32> pc[DEPTH];
#pragma unroll
            for (int k = 0; k < DEPTH; ++k)
                pc[k].fetch(c, PixelAt(c, xy[k0 + k]), pl);
#pragma unroll
            for (int k = 0; k < DEPTH; ++k)
                a = k0 + k == 0 ? pc[k].cost(c) : a + pc[k].cost(c);
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1)
            a = a + __shfl_xor_sync(0xffffffffu, a, off);
        if (lane == 0)
            reinterpret_cast<float *>(c.pc + wi.y)[w] = a;
        return;
    }
    const int q0 = win * PC_CHUNK + w * (32 * COST_SUBS) + lane;
    uint32_t xy[COST_SUBS];
    int n[COST_SUBS];
#pragma unroll
    for (int s = 0; s < COST_SUBS; ++s)
    {
        const int q = q0 + 32 * s;
        xy[s] = q < c.HW ? c.pix[q] : 0u;
        n[s] = q < c.HW ? c.pnode[q] : c.N; // positions past the list form node N
    }
    after_predecessor();
    PlaneCost<F32> pc[COST_SUBS][P];
#pragma unroll
    for (int s = 0; s < COST_SUBS; ++s)
    {
        const int m = min(n[s], c.N - 1); // a position past the list reads the last node's planes and stays unused
        const float4 *src = c.plane + (size_t)(c.clus ? c.clus[m] : m) * K;
        const PixelAt px(c, xy[s]);
#pragma unroll
        for (int p = 0; p < P; ++p)
            pc[s][p].fetch(c, px, src[p]);
    }
    float4 val[COST_SUBS];
    int seg[COST_SUBS];
    unsigned heads[COST_SUBS];
#pragma unroll
    for (int s = 0; s < COST_SUBS; ++s)
    {
        const int prev = __shfl_up_sync(0xffffffffu, n[s], 1);
        heads[s] = __ballot_sync(0xffffffffu, lane == 0 || prev != n[s]);
        seg[s] = 31 - __clz(heads[s] & (0xffffffffu >> (31 - lane)));
        float cc[P];
#pragma unroll
        for (int p = 0; p < P; ++p)
            cc[p] = pc[s][p].cost(c);
        // S1
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
#pragma unroll
            for (int p = 0; p < P; ++p)
            {
                const float u = __shfl_up_sync(0xffffffffu, cc[p], off);
                if (lane - off >= seg[s])
                    cc[p] = u + cc[p];
            }
        val[s] = make_float4(cc[0], cc[1], cc[2], cc[3]);
        const int k = w * COST_SUBS + s;
        if (lane == 0)
            sh.first[k] = n[s];
        if (lane == 31)
        {
            sh.last[k] = n[s];
            sh.whole[k] = seg[s] == 0;
            sh.tail[k] = val[s];
        }
    }
    __syncthreads();
    // S2 and the sums of the segments that end here (a segment at lane 31
    // goes on if the next sub-window starts with its node)
#pragma unroll
    for (int s = 0; s < COST_SUBS; ++s)
    {
        const int k = w * COST_SUBS + s;
        const bool tail = lane == 31 || ((heads[s] >> (lane + 1)) & 1u);
        if (!tail || n[s] >= c.N || (lane == 31 && k + 1 < SUBS && sh.first[k + 1] == n[s]))
            continue;
        if (seg[s] == 0 && k > 0 && sh.last[k - 1] == n[s])
        {
            int j = k - 1; // the sub-window where the node's run inside the window starts
            while (j > 0 && sh.whole[j] && sh.last[j - 1] == n[s])
                --j;
            float4 a = sh.tail[j];
            for (++j; j < k; ++j)
            {
                const float4 u = sh.tail[j];
                a = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, a.w + u.w);
            }
            val[s] = make_float4(a.x + val[s].x, a.y + val[s].y, a.z + val[s].z, a.w + val[s].w);
        }
        c.pc[wi.y + n[s] - wi.x] = val[s];
    }
}

struct CostDesc
{
    int nt;
    int pre[MAXV + 1];
    CostArgs t[MAXV];
};
__global__ void __launch_bounds__(COST_T, COST_MIN_BLOCKS) k_cost(const __grid_constant__ CostDesc d)
{
    __shared__ CostShared sh;
    let_successor_start();
    int ti = 0;
    while (ti + 1 < d.nt && (int)blockIdx.x >= d.pre[ti + 1])
        ++ti;
    const CostArgs &c = d.t[ti];
    const int win = blockIdx.x - d.pre[ti];
    if (c.volf) // uniform per view
        cost_window<true, 4>(c, win, sh);
    else
        cost_window<false, 4>(c, win, sh);
}

// init_bp, continued: the prior planes in every slot group and their costs,
// belief = cost (init_bp + copy_prior_plane, hbp_isp.cu:56-73, :930-950).
__global__ void __launch_bounds__(128) k_init_nodes(const ViewDev *__restrict__ V, StepDesc d)
{
    int item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= d.pre[d.nt])
        return;
    int ti = find_task(d, item);
    const Task &t = d.t[ti];
    const ViewDev &v = *t.vd;
    const LevelDev &l = *t.lvl;
    int n = item - d.pre[ti];
    if (n < l.N)
    {
        const float4 a = sum_chunks(v.b.pc[t.pb], l.chunk_off[n], l.chunk_off[n + 1]);
        float *cs = l.cost + (size_t)n * K;
        float *bl = l.belief + (size_t)n * K;
        cs[0] = cs[4] = a.x;
        cs[1] = cs[5] = a.y;
        cs[2] = cs[6] = a.z;
        cs[3] = cs[7] = a.w;
        for (int k = 0; k < K; ++k)
            bl[k] = cs[k];
        const float4 *pp = t.lvh->plane + (size_t)l.clus[n] * K;
        for (int k = 0; k < K; ++k)
            l.plane[(size_t)n * K + k] = pp[k % P];
    }
}

// passing_msg_k + smooth_msg_k + normalize_msg_k (hbp_isp.cu:273-355): the
// message of edge s -> t for each of s's 12 labels y is the sum over t's two
// label groups of min_q (c0 * min(phi(y, q) / 3 / dist_pos, tau) + mp_q), then
// normalised. min(phi / 3 / dist_pos, tau) is taken as min(phi * rq, tau), rq =
// (1/3) / dist_pos rounded once per edge (the oracle states the same form):
// every label takes the same few instructions, no division and no branch per
// label. phi(y, q) = sum_i |vs_y,i - vt_q,i| over the six points, v = fma(a,
// X_i, fma(b, Y_i, c)).
struct EdgeArgs
{
    const int2 *bd;
    const int *bdl, *rev;
    const float *dc; // 2E: colour weight, centroid distance
    const int4 *pid;
    const float4 *plane;
    const float *belief;
    const unsigned long long *keep;
    const void *msg_in; // the previous step's messages [E][K], float or __half
    void *msg_out;
    int E, fp16, first;
    float tau;
};
struct EdgeDesc
{
    int nt;
    int pre[MAXV + 1]; // blocks before each task
    EdgeArgs t[MAXV];
};
constexpr int EDGE_T = 128, EDGE_LANES = 4;
// Directed edges per fused launch below which each takes eight lanes: they fit
// 48 registers, so ten blocks run on an SM instead of eight and the windows of a
// 720x496 view start together (BP 22.8 -> 22.1 ms, 1440x992 86.4 -> 84.3); above,
// the lanes' repeated work costs more (eight everywhere: 23.0 / 84.5).
constexpr long EIGHT_BELOW = 16384;
constexpr int BOTH_BLOCKS_8 = 10, BOTH_BLOCKS = 8; // of k_cost_edges per SM
// Data-cost windows in flight up to which a step's two kernels are one launch
// (BP ms, one launch / two: 96x64 9.8 / 12.6, 720x496 24.8 / 30.1, four of them
// 65.2 / 67.9, eight 117.8 / 108.9; 1440x992 88.9 / 90.8, two 159.7 / 157.6).
constexpr long BOTH_WINDOWS = 6000;
// Directed edges per launch below which each takes four lanes instead of one
// thread. The lanes repeat the points and the source labels' values (an eighth
// more instructions), so a launch that fills the chip is faster without them
// (1.9M edges: 110 us against 140, 420K: 37 / 41), one that waits for its
// longest chain is faster with them (25K edges: 15.5 / 13.4 us with the
// events' 5; 96x64 pair 23.6 / 22.7 ms).
constexpr long EDGE_LANES_BELOW = 32768;

struct Edge
{
    int2 st;
    int rev;
    float X[6], Y[6]; // the six points, lower-index node's three first (the same order for an edge and its reverse)
    float c0, rq;

    __device__ __forceinline__ Edge(const EdgeArgs &t, int e)
    {
        st = t.bd[e];
        c0 = fmaxf(t.dc[e], 0.01f) * (float)t.bdl[e];
        rq = (1.0f / 3.0f) / fmaxf(t.dc[t.E + e], 1.0f);
        rev = t.rev[e];
        after_predecessor();
        const int4 a = t.pid[min(st.x, st.y)], b = t.pid[max(st.x, st.y)];
        const uint32_t pts[6] = {(uint32_t)a.x, (uint32_t)a.y, (uint32_t)a.z, (uint32_t)b.x, (uint32_t)b.y, (uint32_t)b.z};
#pragma unroll
        for (int i = 0; i < 6; ++i)
        {
            X[i] = (float)px_x(pts[i]);
            Y[i] = (float)px_y(pts[i]);
        }
    }
    __device__ __forceinline__ float at(float4 pl, int i) const { return __fmaf_rn(pl.x, X[i], __fmaf_rn(pl.y, Y[i], pl.z)); }
};

// t's belief of label p without s's last message to it (ping_pang_msg +
// select_msg: that message's slot is where p stood before the select)
__device__ __forceinline__ float passed(const EdgeArgs &t, float belief, unsigned long long kl, size_t rev, int p)
{
    const int slot = p < (int)(kl & 15ull) ? (int)((kl >> (4 + 4 * p)) & 15ull) : p;
    const size_t i = rev * K + slot;
    return belief - (t.fp16 ? __half2float(static_cast<const __half *>(t.msg_in)[i]) : static_cast<const float *>(t.msg_in)[i]);
}

// T labels of one group: the smallest c0 * min(phi * rq, tau) + mp. A
// NaN never wins, as in a chain of m < mn from FLT_MAX.
template <int T>
__device__ __forceinline__ float group_min(const EdgeArgs &t, const Edge &g, const float phi[T], const float mp[T])
{
    float mn = FLT_MAX;
#pragma unroll
    for (int k = 0; k < T; ++k)
        mn = fminf(mn, __fmaf_rn(g.c0, fminf(phi[k] * g.rq, t.tau), mp[k]));
    return mn;
}

// Normalisation: the reference subtracts the mean (normalize_msg_k); FP16
// storage subtracts the message's minimum instead, so the stored values start
// at 0 and keep FP16's relative precision (the beliefs of a node shift by a
// per-message constant, which leaves their order unchanged).

// LANES lanes per edge, four or eight: h halves the source labels (6h ..
// 6h+5), g is the target group, and of eight lanes u takes two of its four
// labels.
template <int LANES>
__device__ __forceinline__ void edge_lanes(const EdgeArgs &t, int e, int le)
{
    if (e >= t.E) // uniform over the edge's lanes
        return;
    constexpr int T = 2 * K / 3 / (LANES / 2); // target labels of a lane: 4 or 2
    const unsigned gm = (LANES == 8 ? 0xffu : 0xfu) << (threadIdx.x & (32 - LANES));
    const int g = le & 1, u = LANES == 8 ? (le >> 1) & 1 : 0, h = le / (LANES / 2);
    const int q0 = g * P + u * T;
    const Edge ed(t, e);
    float mp[T];
    if constexpr (T == 4)
    {
        const float4 b = *reinterpret_cast<const float4 *>(t.belief + (size_t)ed.st.y * K + q0);
        mp[0] = b.x, mp[1] = b.y, mp[2] = b.z, mp[3] = b.w;
    }
    else
    {
        const float2 b = *reinterpret_cast<const float2 *>(t.belief + (size_t)ed.st.y * K + q0);
        mp[0] = b.x, mp[1] = b.y;
    }
    if (!t.first)
    {
        const unsigned long long kl = t.keep[ed.st.y];
#pragma unroll
        for (int k = 0; k < T; ++k)
            mp[k] = passed(t, mp[k], kl, (size_t)ed.rev, q0 + k);
    }
    float vt[T][6];
#pragma unroll
    for (int k = 0; k < T; ++k)
    {
        const float4 tp = t.plane[(size_t)ed.st.y * K + q0 + k];
#pragma unroll
        for (int i = 0; i < 6; ++i)
            vt[k][i] = ed.at(tp, i);
    }
    float out[K / 2];
#pragma unroll
    for (int j = 0; j < K / 2; ++j)
    {
        const float4 ps = t.plane[(size_t)ed.st.x * K + h * (K / 2) + j];
        float phi[T];
#pragma unroll
        for (int i = 0; i < 6; ++i)
        {
            const float vs = ed.at(ps, i);
#pragma unroll
            for (int k = 0; k < T; ++k)
                phi[k] = i == 0 ? fabsf(vs - vt[k][0]) : phi[k] + fabsf(vs - vt[k][i]);
        }
        float mine = group_min<T>(t, ed, phi, mp);
        if (LANES == 8)
            mine = fminf(mine, __shfl_xor_sync(gm, mine, 2));
        const float other = __shfl_xor_sync(gm, mine, 1);
        out[j] = (0.f + (g ? other : mine)) + (g ? mine : other); // group 0's first, as the reference
    }
    float norm;
    if (t.fp16)
    {
        norm = out[0];
#pragma unroll
        for (int j = 1; j < K / 2; ++j)
            norm = fminf(norm, out[j]);
        norm = fminf(norm, __shfl_xor_sync(gm, norm, LANES / 2));
    }
    else
    {
        // the sum over the 12 labels in order: labels 0-5, carried on by h = 1
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < K / 2; ++j)
            s = s + out[j];
        s = __shfl_xor_sync(gm, s, LANES / 2);
#pragma unroll
        for (int j = 0; j < K / 2; ++j)
            s = s + out[j];
        norm = __shfl_sync(gm, s, LANES / 2 + g, LANES) / (float)K; // h = 1's
    }
    if (u)
        return;
    const size_t o = (size_t)e * K + h * (K / 2) + g * (K / 4);
#pragma unroll
    for (int j = 0; j < K / 4; ++j)
    {
        const float v = (g ? out[K / 4 + j] : out[j]) - norm;
        if (t.fp16)
            static_cast<__half *>(t.msg_out)[o + j] = __float2half_rn(v);
        else
            static_cast<float *>(t.msg_out)[o + j] = v;
    }
}

__device__ __forceinline__ int edge_task(const EdgeDesc &d)
{
    int k = 0;
    while (k + 1 < d.nt && (int)blockIdx.x >= d.pre[k + 1])
        ++k;
    return k;
}

__global__ void __launch_bounds__(EDGE_T) k_edges_lanes(const __grid_constant__ EdgeDesc d)
{
    let_successor_start();
    const int ti = edge_task(d);
    edge_lanes<EDGE_LANES>(d.t[ti], (blockIdx.x - d.pre[ti]) * (EDGE_T / EDGE_LANES) + threadIdx.x / EDGE_LANES, threadIdx.x % EDGE_LANES);
}

// message e's 12 values; FP16 storage rounds each to nearest, the arithmetic
// on messages is FP32 either way
__device__ __forceinline__ void store_msg(const EdgeArgs &t, size_t e, const float v[K])
{
    if (t.fp16)
    {
        uint2 *h = static_cast<uint2 *>(t.msg_out) + e * (K / 4);
#pragma unroll
        for (int i = 0; i < K / 4; ++i)
        {
            __half2 lo = __floats2half2_rn(v[4 * i], v[4 * i + 1]);
            __half2 hi = __floats2half2_rn(v[4 * i + 2], v[4 * i + 3]);
            h[i] = make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
        }
    }
    else
    {
        float4 *o = static_cast<float4 *>(t.msg_out) + e * (K / 4);
#pragma unroll
        for (int i = 0; i < K / 4; ++i)
            o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
}

// One thread per edge: the eight target labels' point values are held in
// registers (96 registers, 5 blocks of 128 per SM; splitting the two label
// groups into two passes fits 7 blocks but reloads every source plane and
// measured 4% slower).
__global__ void __launch_bounds__(EDGE_T, 5) k_edges(const __grid_constant__ EdgeDesc d)
{
    __shared__ float s_out[K][EDGE_T];
    let_successor_start();
    const int ti = edge_task(d);
    const EdgeArgs &t = d.t[ti];
    const int e = (blockIdx.x - d.pre[ti]) * EDGE_T + threadIdx.x;
    if (e >= t.E)
        return;
    const Edge ed(t, e);
    const float *bt = t.belief + (size_t)ed.st.y * K;
    float mp[2][P];
#pragma unroll
    for (int p = 0; p < 2 * P; ++p)
        mp[p / P][p % P] = bt[p];
    if (!t.first)
    {
        const unsigned long long kl = t.keep[ed.st.y];
#pragma unroll
        for (int p = 0; p < 2 * P; ++p)
            mp[p / P][p % P] = passed(t, mp[p / P][p % P], kl, (size_t)ed.rev, p);
    }
    float vt[2][P][6];
#pragma unroll
    for (int k = 0; k < 2 * P; ++k)
    {
        const float4 tp = t.plane[(size_t)ed.st.y * K + k];
#pragma unroll
        for (int i = 0; i < 6; ++i)
            vt[k / P][k % P][i] = ed.at(tp, i);
    }
    float sum = 0.f;
#pragma unroll 1
    for (int y = 0; y < K; ++y)
    {
        const float4 ps = t.plane[(size_t)ed.st.x * K + y];
        float phi[2][P];
#pragma unroll
        for (int i = 0; i < 6; ++i)
        {
            const float vs = ed.at(ps, i);
#pragma unroll
            for (int k = 0; k < 2 * P; ++k)
                phi[k / P][k % P] = i == 0 ? fabsf(vs - vt[k / P][k % P][0]) : phi[k / P][k % P] + fabsf(vs - vt[k / P][k % P][i]);
        }
        const float acc = (0.f + group_min<P>(t, ed, phi[0], mp[0])) + group_min<P>(t, ed, phi[1], mp[1]);
        s_out[y][threadIdx.x] = acc;
        sum = sum + acc;
    }
    float out[K];
#pragma unroll
    for (int y = 0; y < K; ++y)
        out[y] = s_out[y][threadIdx.x];
    float norm = sum / (float)K;
    if (t.fp16)
    {
        norm = out[0];
#pragma unroll
        for (int k = 1; k < K; ++k)
            norm = fminf(norm, out[k]);
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        out[k] = out[k] - norm;
    store_msg(t, (size_t)e, out);
}

// Data cost and edge messages of a step in one launch: neither reads what the
// other writes (the messages use the selected planes and beliefs, not the
// candidates' costs). A task's blocks alternate between windows and edges, so
// that the volume reads of one wait beside the arithmetic of the other.
struct StepArgs
{
    CostArgs cost;
    EdgeArgs edge;
    int windows, edge_blocks;
};
struct BothDesc
{
    int nt;
    int pre[MAXV + 1]; // blocks before each task
    StepArgs t[MAXV];
};
static_assert(COST_T == EDGE_T, "one block shape for both");
template <int LANES>
__global__ void __launch_bounds__(EDGE_T, LANES == 8 ? BOTH_BLOCKS_8 : BOTH_BLOCKS) k_cost_edges(const __grid_constant__ BothDesc d)
{
    __shared__ CostShared sh;
    let_successor_start();
    int ti = 0;
    while (ti + 1 < d.nt && (int)blockIdx.x >= d.pre[ti + 1])
        ++ti;
    const StepArgs &t = d.t[ti];
    const int b = blockIdx.x - d.pre[ti], paired = min(t.windows, t.edge_blocks);
    const bool edges = b < 2 * paired ? (b & 1) == 0 : t.edge_blocks > t.windows;
    const int item = b < 2 * paired ? b >> 1 : b - paired;
    if (edges)
        edge_lanes<LANES>(t.edge, item * (EDGE_T / LANES) + threadIdx.x / LANES, threadIdx.x % LANES);
    else if (t.cost.volf) // uniform per view
        cost_window<true, 8>(t.cost, item, sh);
    else
        cost_window<false, 8>(t.cost, item, sh);
}

// map_msg (hbp_isp.cu:783-841), one warp per node of the task's level; into
// the view's disparity/planes, or (MAP_LEVEL) into the per-level maps of
// run_ms_vis (hbp_isp.cu:1348-1383)
constexpr int MAP_LEVEL = 1;
__global__ void __launch_bounds__(128) k_map(const ViewDev *__restrict__ V, StepDesc d)
{
    const int lane = threadIdx.x & 31;
    const int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (item >= d.pre[d.nt])
        return;
    int ti = find_task(d, item);
    const Task &t = d.t[ti];
    const ViewDev &v = *t.vd;
    const LevelDev &l = *t.lvl;
    const Common &c = v.c;
    int n = item - d.pre[ti];
    const float *bl = l.belief + (size_t)n * K;
    float mn = bl[0];
    for (int p = 1; p < P; ++p)
        mn = fminf(mn, bl[p]);
    int mp = 0;
    for (int p = 0; p < P; ++p)
        if (bl[p] == mn)
        {
            mp = p;
            break;
        }
    float4 pl = l.plane[(size_t)n * K + mp];
    float *disp = v.disp, *plane_out = v.plane_out;
    if (t.mode == MAP_LEVEL)
    {
        const size_t off = (size_t)(v.L - 1 - t.li) * c.W * c.H;
        disp = v.lvl_disp + off;
        plane_out = v.lvl_plane ? v.lvl_plane + 3 * off : nullptr;
    }
    for (int j = l.pix_off[n] + lane; j < l.pix_off[n + 1]; j += 32)
    {
        uint32_t xy = l.pix[j];
        int x = px_x(xy), y = px_y(xy);
        float dd = pl.x * (float)x + pl.y * (float)y + pl.z;
        dd = fminf(fmaxf(dd, 0.f), (float)(c.D - 1));
        size_t id = (size_t)y * c.W + x;
        disp[id] = dd;
        if (plane_out)
        {
            plane_out[3 * id] = pl.x;
            plane_out[3 * id + 1] = pl.y;
            plane_out[3 * id + 2] = pl.z;
        }
    }
}

inline int blocks(long n, int t) { return ceil_div(n, t); }

} // namespace

// ---------------------------------------------------------------------------
// host side
struct ViewPlan::Impl
{
    ViewDev vd;              // host copy
    ViewDev *vd_dev = nullptr; // the same record in device memory
    std::vector<LevelDev> lv;
};

ViewPlan::ViewPlan() : impl(new Impl) {}
ViewPlan::~ViewPlan() { delete impl; }

// Per-level setup of one view (HBP_ISP constructor and the first loop of
// run_ms: setup_D4, reverse_bd_id, compute_dist_color_pos, sort_clus;
// hbp_isp.cu:871-891, :952-1019), the BP buffers, and the view descriptor.
// Persistent data go to `persist`, sort/scan temporaries to `tmp`.
void hbp_prepare(const Pyramid &pyr, const CostVolume &cv, const float *wta, int D,
                 const HbpParams &prm, float *disp, float *plane_out, Arena &persist, Arena &tmp,
                 cudaStream_t st, ViewPlan &vp)
{
    if ((cv.u8 != nullptr) == (cv.f32 != nullptr) || !(cv.tau > 0.0f))
        throw StatusError{HBP_ERR_INVALID_ARG, "exactly one cost volume (uint8 or float) and tau > 0"};
    const int L = pyr.L, W = pyr.W, H = pyr.H, HW = W * H;
    const int m = prm.min_level;
    if (L < 1 || m < 0 || m > L - 1)
        throw StatusError{HBP_ERR_INVALID_ARG, "min_level must lie in [0, levels-1]"};
    if ((int)pyr.N.size() != L || (int)pyr.E.size() != L || (int)pyr.node_off.size() != L ||
        (int)pyr.edge_off.size() != L || (int)pyr.child_base.size() != L || (int)pyr.nb_base.size() != L)
        throw StatusError{HBP_ERR_INTERNAL, "pyramid bookkeeping inconsistent"};
    Common c{W, H, D, ceil_div(W, VT_W), prm.alpha, cv.tau, prm.tau_smooth, cv.u8, cv.f32, wta};
    std::vector<LevelDev> &lv = vp.impl->lv;
    lv.assign(L, LevelDev{});
    vp.L = L;
    vp.min_level = m;
    vp.D = D;
    vp.HW = HW;
    vp.levelN.assign(L, 0);
    vp.levelE.assign(L, 0);
    vp.levelC.assign(L, 0);
    int Nmax = 1, Emax = 1, CHmax = 1;
    size_t tm = tmp.mark();
    int *im = tmp.alloc<int>(HW), *im2 = tmp.alloc<int>(HW);
    uint32_t *ka = tmp.alloc<uint32_t>(HW), *va = tmp.alloc<uint32_t>(HW);
    int *cnt = tmp.alloc<int>(HW + 1);
    iota_int<<<blocks(HW, 256), 256, 0, st>>>(im, HW);
    note_launch();
    HBP_LAUNCH_CHECK();
    for (int l = 0; l < L; ++l)
    {
        LevelDev &d = lv[l];
        d.N = pyr.N[l];
        d.E = pyr.E[l];
        d.Nh = l + 1 < L ? pyr.N[l + 1] : 1;
        d.clus = pyr.clus + pyr.node_off[l];
        d.bd = pyr.bd + pyr.edge_off[l];
        d.bdl = pyr.bdl + pyr.edge_off[l];
        d.nb_off = pyr.nb_off + pyr.nb_base[l];
        d.child = pyr.child + pyr.node_off[l];
        d.child_off = pyr.child_off + pyr.child_base[l];
        vp.levelN[l] = d.N;
        vp.levelE[l] = d.E;
        if (l >= m)
        {
            const int N = d.N, E = d.E;
            uint32_t *pix = persist.alloc<uint32_t>(HW);
            int *pix_off = persist.alloc<int>(N + 1);
            int *pnode = persist.alloc<int>(HW); // the sorted keys
            uint32_t *key = reinterpret_cast<uint32_t *>(pnode);
            iota_xy<<<blocks(HW, 256), 256, 0, st>>>(key, pix, im, W, HW);
            note_launch();
            HBP_LAUNCH_CHECK();
            int bits = 1;
            while ((1 << bits) < N)
                ++bits;
            radix_sort_pairs_u32(key, pix, ka, va, HW, bits, tmp, st);
            run_starts<<<blocks(HW, 256), 256, 0, st>>>(key, HW, N, pix_off);
            note_launch();
            HBP_LAUNCH_CHECK();
            int *chunk_off = persist.alloc<int>(N + 1);
            chunk_counts<<<blocks(N + 1, 256), 256, 0, st>>>(pix_off, N, cnt);
            note_launch();
            exclusive_scan(cnt, chunk_off, N + 1, nullptr, tmp, st);
            // a node's chunks are the windows it overlaps: at most one more per
            // node but the first than there are windows
            const int nwin = ceil_div(HW, PC_CHUNK);
            d.nchunks = nwin + N - 1;
            vp.levelC[l] = d.nchunks;
            int2 *win = persist.alloc<int2>(nwin);
            window_info<<<blocks(nwin, 256), 256, 0, st>>>(key, pix_off, chunk_off, HW, win);
            note_launch();
            HBP_LAUNCH_CHECK();
            int *rev = persist.alloc<int>(E);
            reverse_ids<<<blocks(E, 256), 256, 0, st>>>(d.bd, d.nb_off, E, rev);
            note_launch();
            float *ml = tmp.alloc<float>(3 * (size_t)N), *mx = persist.alloc<float>(N), *my = persist.alloc<float>(N);
            level_means<<<blocks(N, 256), 256, 0, st>>>(pyr.sums + 6 * pyr.node_off[l], N, mx, my, ml);
            note_launch();
            float *dc = persist.alloc<float>(2 * (size_t)E);
            edge_weights<<<blocks(E, 256), 256, 0, st>>>(d.bd, E, N, ml, mx, my, dc);
            note_launch();
            HBP_LAUNCH_CHECK();
            d.pix = pix;
            d.pix_off = pix_off;
            d.chunk_off = chunk_off;
            d.pnode = pnode;
            d.win = win;
            d.rev = rev;
            d.dc = dc;
            d.mx = mx;
            d.my = my;
            // one fill for the level's node records, which lie side by side
            d.plane = persist.alloc<float4>((size_t)N * K);
            d.cost = persist.alloc<float>((size_t)N * K);
            d.belief = persist.alloc<float>((size_t)N * K);
            d.pid = persist.alloc<int4>(N);
            d.keep = persist.alloc<unsigned long long>(N);
            HBP_CUDA(cudaMemsetAsync(d.plane, 0, (size_t)(reinterpret_cast<char *>(d.keep + N) - reinterpret_cast<char *>(d.plane)), st));
            Nmax = std::max(Nmax, N);
            Emax = std::max(Emax, E);
            CHmax = std::max(CHmax, d.nchunks);
        }
        if (l + 1 < L)
        {
            compose_im_clus<<<blocks(HW, 256), 256, 0, st>>>(im, d.clus, HW, im2);
            note_launch();
            HBP_LAUNCH_CHECK();
            std::swap(im, im2);
        }
    }
    ViewDev &vd = vp.impl->vd;
    vd.c = c;
    vd.b.fp16 = prm.msg_fp16 ? 1 : 0;
    vd.L = L;
    LevelDev *lv_dev = persist.alloc<LevelDev>(L);
    HBP_CUDA(cudaMemcpyAsync(lv_dev, lv.data(), sizeof(LevelDev) * L, cudaMemcpyHostToDevice, st));
    vd.lv = lv_dev;
    for (int k = 0; k < 2; ++k)
    {
        vd.b.msgt[k] = prm.msg_fp16 ? (void *)persist.alloc<__half>((size_t)Emax * K)
                                    : (void *)persist.alloc<float>((size_t)Emax * K);
        vd.b.pc[k] = persist.alloc<float4>(CHmax);
    }
    vd.disp = disp;
    vd.plane_out = plane_out;
    vd.lvl_disp = prm.level_disp;
    vd.lvl_plane = prm.level_disp ? prm.level_plane : nullptr;
    vp.levels = prm.level_disp != nullptr;
    vp.impl->vd_dev = persist.alloc<ViewDev>(1);
    HBP_CUDA(cudaMemcpyAsync(vp.impl->vd_dev, &vd, sizeof(ViewDev), cudaMemcpyHostToDevice, st));
    HBP_CUDA(cudaStreamSynchronize(st)); // lv and vd (host) feed the copies above
    tmp.rewind(tm);
}

namespace
{
enum Phase
{
    PH_INIT,  // level setup: priors, their costs, beliefs (init_bp)
    PH_STEP,  // one candidate step + data cost + BP sweep
    PH_FINAL, // the level's last select
    PH_MAP_LEVEL, // map_msg of level li into the per-level maps (run_ms_vis)
    PH_MAP,   // map_msg at min_level
    PH_DONE
};

} // namespace

// One view's place in HBP_ISP::run_ms (hbp_isp.cu:1313-1346): level li, outer
// iteration i, candidate step it (0-3 RANSAC, 4 spatial, 5 random adjust).
struct BpScheduler::View
{
    ViewPlan *vp;
    void *user;
    int phase = PH_INIT, li = 0, i = 0, it = 0, step = 0;
    LcgJump drawn{0};   // the level's draws so far (NodeArgs::seed_a, seed_c)
    LcgJump spatial{0}; // and the spatial steps' (SpatialArgs::seed_a, seed_c)
    float max_dz = 0, max_dn = 0;

    int iter_bp() const { return 10 + 10 * li; }
    void enter_level(int level)
    {
        li = level;
        phase = PH_INIT;
        step = 0;
        i = 0;
        it = 0;
        drawn = spatial = LcgJump(0);
        max_dz = (float)vp->D / 2.0f * (float)li / (float)vp->L;
        max_dn = 1.0f * (float)li / (float)vp->L;
    }
    // skip random-adjust steps that do not apply; end the level after its
    // last iteration
    void settle()
    {
        while (phase == PH_STEP)
        {
            if (i >= iter_bp())
            {
                phase = PH_FINAL;
                break;
            }
            if (it == 5 && !(i > iter_bp() / 4 * 3 && max_dz >= 0.01f))
            {
                it = 0;
                ++i;
                continue;
            }
            break;
        }
    }
    int kind() const { return it <= 3 ? 0 : it == 4 ? 1 : 2; }
};

struct BpScheduler::Impl
{
    HbpParams prm;
    cudaStream_t st;
    std::vector<View> views;
    long ticks = 0;

    Task task_of(const View &v, bool first, int pb, int mode) const
    {
        const ViewPlan &vp = *v.vp;
        const ViewDev &vd = vp.impl->vd;
        Task t{};
        t.vd = vp.impl->vd_dev;
        t.lvl = vd.lv + v.li;
        t.lvh = v.li + 1 < vp.L ? vd.lv + v.li + 1 : t.lvl;
        t.v = 0;
        t.li = v.li;
        t.first = first ? 1 : 0;
        t.pb = pb;
        t.mb = v.step & 1;
        t.mode = mode;
        return t;
    }
    static CostArgs cost_args(const View &v, const Task &s, int mode)
    {
        const ViewDev &vd = v.vp->impl->vd;
        const LevelDev &l = v.vp->impl->lv[v.li];
        const bool init = mode == COST_INIT;
        return CostArgs{l.pix, l.pnode, l.win, init ? v.vp->impl->lv[v.li + 1].plane : l.plane + 2 * P, init ? l.clus : nullptr,
                        vd.b.pc[s.pb], vd.c.vol, vd.c.volf, vd.c.W * vd.c.H, l.N, vd.c.TX, vd.c.D, vd.c.lambda, vd.c.tau};
    }
    static int windows(const View &v) { return ceil_div(v.vp->HW, PC_CHUNK); }
    static EdgeArgs edge_args(const View &v, const Task &s)
    {
        const ViewDev &vd = v.vp->impl->vd;
        const LevelDev &l = v.vp->impl->lv[v.li];
        return EdgeArgs{l.bd, l.bdl, l.rev, l.dc, l.pid, l.plane, l.belief, l.keep, vd.b.msgt[s.mb ^ 1],
                        vd.b.msgt[s.mb], l.E, vd.b.fp16, s.first, vd.c.tau_smooth};
    }
    // Data cost of the tasks, a block per window: of the parents' best planes
    // (COST_INIT) or of the candidates, in descriptors of at most MAXV views.
    template <typename F>
    void launch_cost(const std::vector<const View *> &vs, const std::vector<Task> &ts, int mode, F &&f)
    {
        for (size_t b = 0; b < ts.size(); b += MAXV)
        {
            CostDesc d;
            d.nt = (int)std::min<size_t>(MAXV, ts.size() - b);
            d.pre[0] = 0;
            for (int k = 0; k < d.nt; ++k)
            {
                d.t[k] = cost_args(*vs[b + k], ts[b + k], mode);
                d.pre[k + 1] = d.pre[k] + windows(*vs[b + k]);
            }
            f([&] { launch_chained(k_cost, d.pre[d.nt], COST_T, st, d); });
        }
    }
    // Data cost of the candidates and edge messages of the tasks in one launch
    // per MAXV views.
    template <typename F>
    void launch_both(const std::vector<const View *> &vs, const std::vector<Task> &ts, bool few, F &&f)
    {
        const int lanes = few ? 8 : EDGE_LANES;
        for (size_t b = 0; b < ts.size(); b += MAXV)
        {
            BothDesc d;
            d.nt = (int)std::min<size_t>(MAXV, ts.size() - b);
            d.pre[0] = 0;
            for (int k = 0; k < d.nt; ++k)
            {
                StepArgs &t = d.t[k];
                t.cost = cost_args(*vs[b + k], ts[b + k], COST_STEP);
                t.edge = edge_args(*vs[b + k], ts[b + k]);
                t.windows = windows(*vs[b + k]);
                t.edge_blocks = ceil_div(t.edge.E, EDGE_T / lanes);
                d.pre[k + 1] = d.pre[k] + t.windows + t.edge_blocks;
            }
            f([&] { launch_chained(few ? k_cost_edges<8> : k_cost_edges<EDGE_LANES>, d.pre[d.nt], EDGE_T, st, d); });
        }
    }
    // Node phase of the tasks.
    template <typename F>
    void launch_node(const std::vector<const View *> &vs, const std::vector<Task> &ts, F &&f)
    {
        for (size_t b = 0; b < ts.size(); b += MAXV)
        {
            NodeDesc d;
            d.nt = (int)std::min<size_t>(MAXV, ts.size() - b);
            bool blocks_of_nodes = false;
            long nodes = 0;
            for (int k = 0; k < d.nt; ++k)
                nodes += vs[b + k]->vp->levelN[vs[b + k]->li];
            d.pre[0] = 0;
            for (int k = 0; k < d.nt; ++k)
            {
                const View &v = *vs[b + k];
                const Task &s = ts[b + k];
                const ViewDev &vd = v.vp->impl->vd;
                const LevelDev &l = v.vp->impl->lv[v.li];
                NodeArgs &t = d.t[k];
                t.nb_off = l.nb_off;
                t.chunk_off = l.chunk_off;
                t.pix_off = l.pix_off;
                t.pc = vd.b.pc[s.pb ^ 1];
                t.msg = vd.b.msgt[s.mb ^ 1];
                t.plane = l.plane;
                t.cost = l.cost;
                t.belief = l.belief;
                t.pid = l.pid;
                t.keep = l.keep;
                t.pix = l.pix;
                t.wta = vd.c.wta;
                t.mx = l.mx;
                t.my = l.my;
                t.N = l.N;
                t.W = vd.c.W;
                t.fp16 = vd.b.fp16;
                t.first = s.first;
                t.mode = s.mode;
                t.block_per_node = nodes <= NODE_BLOCK_NODES || l.nchunks >= NODE_BLOCK_CHUNKS * (long)l.N;
                t.seed_a = v.drawn.a;
                t.seed_c = v.drawn.c;
                t.max_dz = v.max_dz;
                t.max_dn = v.max_dn;
                blocks_of_nodes = blocks_of_nodes || t.block_per_node;
                d.pre[k + 1] = d.pre[k] + (t.block_per_node ? l.N : ceil_div(l.N, NODE_PER_BLOCK));
            }
            f([&] { launch_chained(k_node, d.pre[d.nt], NODE_T, st, d, blocks_of_nodes ? NODE_SMEM : 0); });
        }
    }
    // Spatial candidates of the views.
    template <typename F>
    void launch_spatial(const std::vector<const View *> &vs, F &&f)
    {
        for (size_t b = 0; b < vs.size(); b += MAXV)
        {
            SpatialDesc d;
            d.nt = (int)std::min<size_t>(MAXV, vs.size() - b);
            d.pre[0] = 0;
            for (int k = 0; k < d.nt; ++k)
            {
                const View &v = *vs[b + k];
                const LevelDev &l = v.vp->impl->lv[v.li], &h = v.vp->impl->lv[v.li + 1];
                d.t[k] = SpatialArgs{l.clus, l.nb_off, h.nb_off, h.bd, l.child, l.child_off, l.plane, l.N, v.spatial.a, v.spatial.c};
                d.pre[k + 1] = d.pre[k] + ceil_div((long)l.N * P, SPATIAL_T);
            }
            f([&] { launch_chained(k_spatial, d.pre[d.nt], SPATIAL_T, st, d); });
        }
    }
    // Edge messages of the tasks.
    template <typename F>
    void launch_edges(const std::vector<const View *> &vs, const std::vector<Task> &ts, F &&f)
    {
        for (size_t b = 0; b < ts.size(); b += MAXV)
        {
            EdgeDesc d;
            d.nt = (int)std::min<size_t>(MAXV, ts.size() - b);
            long edges = 0;
            for (int k = 0; k < d.nt; ++k)
                edges += vs[b + k]->vp->levelE[vs[b + k]->li];
            const bool lanes = edges < EDGE_LANES_BELOW;
            d.pre[0] = 0;
            for (int k = 0; k < d.nt; ++k)
            {
                d.t[k] = edge_args(*vs[b + k], ts[b + k]);
                d.pre[k + 1] = d.pre[k] + ceil_div(d.t[k].E, lanes ? EDGE_T / EDGE_LANES : EDGE_T);
            }
            if (d.pre[d.nt] == 0)
                continue;
            f([&] { launch_chained(lanes ? k_edges_lanes : k_edges, d.pre[d.nt], EDGE_T, st, d); });
        }
    }
    // Launch f(desc) over the tasks' nodes in descriptors of at most MAXV tasks.
    template <typename F>
    void launch(const std::vector<const View *> &vs, const std::vector<Task> &ts, F &&f)
    {
        for (size_t b = 0; b < ts.size(); b += MAXV)
        {
            StepDesc d{};
            d.nt = (int)std::min<size_t>(MAXV, ts.size() - b);
            d.pre[0] = 0;
            for (int k = 0; k < d.nt; ++k)
            {
                d.t[k] = ts[b + k];
                d.pre[k + 1] = d.pre[k] + vs[b + k]->vp->levelN[vs[b + k]->li];
            }
            if (d.pre[d.nt] > 0)
                f(d);
        }
    }
};

BpScheduler::BpScheduler(const HbpParams &prm, cudaStream_t st) : impl(new Impl)
{
    impl->prm = prm;
    impl->st = st;
}

BpScheduler::~BpScheduler() { delete impl; }

int BpScheduler::active() const { return (int)impl->views.size(); }

long BpScheduler::windows() const
{
    long w = 0;
    for (const View &v : impl->views)
        w += Impl::windows(v);
    return w;
}

void BpScheduler::add(ViewPlan *vp, void *user)
{
    View v;
    v.vp = vp;
    v.user = user;
    if (vp->L - 2 >= vp->min_level)
    {
        if (vp->levels)
        {
            v.li = vp->L - 1; // run_ms_vis maps the top level before any BP
            v.phase = PH_MAP_LEVEL;
        }
        else
            v.enter_level(vp->L - 2);
    }
    else
    {
        v.li = vp->min_level;
        v.phase = PH_MAP;
    }
    impl->views.push_back(v);
}

// One tick: every active view takes one action; one launch per kernel kind
// (per MAXV views) serves all of them. Views never read one another's data, so
// a view's results do not depend on what else is in flight.
void BpScheduler::tick(std::vector<void *> &finished, long windows_in_flight)
{
    Impl &I = *impl;
    const cudaStream_t st = I.st;
    KernelProf *prof = I.prm.prof && I.prm.prof->on ? I.prm.prof : nullptr;
    KernelProf *bprof = prof && prof->breakdown ? prof : nullptr;
    const long tk = I.ticks++;
    const bool sample = bprof && tk % 8 == 0;
    auto run = [&](int kind, int li, auto &&f) {
        if (!bprof)
        {
            f();
            return;
        }
        const int tag = kind * KernelProf::LEVELS + std::min(li, KernelProf::LEVELS - 1);
        bprof->count[tag]++;
        if (sample)
        {
            bprof->markb(st);
            f();
            bprof->markb(st);
            bprof->tagb.push_back(tag);
        }
        else
            f();
    };

    std::vector<const View *> vi, vn, vs, vc, vm;
    std::vector<Task> ti, tn, tc, tm;
    for (const View &v : I.views)
    {
        const bool first = v.step == 0;
        const int pb = v.step & 1;
        switch (v.phase)
        {
        case PH_INIT:
            vi.push_back(&v);
            ti.push_back(I.task_of(v, true, 0, NODE_SELECT));
            break;
        case PH_STEP:
        {
            const int k = v.kind();
            const int mode = k == 0 ? NODE_SELECT_RANSAC : k == 2 ? NODE_SELECT_RANDOM : NODE_SELECT;
            vn.push_back(&v);
            tn.push_back(I.task_of(v, first, pb, mode));
            if (k == 1)
                vs.push_back(&v);
            vc.push_back(&v);
            tc.push_back(I.task_of(v, first, pb, mode));
            break;
        }
        case PH_FINAL:
            vn.push_back(&v);
            tn.push_back(I.task_of(v, false, pb, NODE_SELECT));
            break;
        case PH_MAP_LEVEL:
            vm.push_back(&v);
            tm.push_back(I.task_of(v, false, pb, MAP_LEVEL));
            break;
        case PH_MAP:
            vm.push_back(&v);
            tm.push_back(I.task_of(v, false, pb, NODE_SELECT));
            if (v.vp->levels)
            {
                vm.push_back(&v);
                tm.push_back(I.task_of(v, false, pb, MAP_LEVEL));
            }
            break;
        }
    }
    // NVTX range named after the pyramid level of the tick's first view (the
    // profiling recipes select one level of a lockstep batch with it)
    char rname[32];
    std::snprintf(rname, sizeof(rname), "bp_level_%d", I.views.empty() ? -1 : I.views[0].li);
    NvtxRange tick_range(rname);
    const int lvl_i = vi.empty() ? 0 : vi[0]->li, lvl_n = vn.empty() ? 0 : vn[0]->li;
    const int lvl_c = vc.empty() ? 0 : vc[0]->li, lvl_s = vs.empty() ? 0 : vs[0]->li;
    // level setup (init_bp): prior costs into pc[0], then planes, costs, beliefs
    I.launch_cost(vi, ti, COST_INIT, [&](auto &&go) { run(6, lvl_i, go); });
    I.launch(vi, ti, [&](const StepDesc &d) {
        run(7, lvl_i, [&] { k_init_nodes<<<blocks(d.pre[d.nt], 128), 128, 0, st>>>(nullptr, d); });
        note_launch();
    });
    // node phase: select of the previous step + the step's candidates
    I.launch_node(vn, tn, [&](auto &&go) { run(0, lvl_n, go); });
    // spatial candidates
    I.launch_spatial(vs, [&](auto &&go) { run(3, lvl_s, go); });
    // data cost of the candidates and the BP sweep
    const bool tp = prof && !vc.empty() && (tk % 16 == 0);
    long step_edges = 0;
    for (const View *v : vc)
        step_edges += v->vp->levelE[v->li];
    if (windows_in_flight <= BOTH_WINDOWS && !tp) // a step of the per-kernel timing issues the two by themselves
    {
        I.launch_both(vc, tc, step_edges < EIGHT_BELOW, [&](auto &&go) { run(9, lvl_c, go); });
        vc.clear();
        tc.clear();
    }
    I.launch_cost(vc, tc, COST_STEP, [&](auto &&go) {
        run(4, lvl_c, [&] {
            if (tp)
                prof->mark(st);
            go();
            if (tp)
                prof->mark(st);
        });
    });
    if (tp)
    {
        // compulsory bytes of the timed data-cost launches: every pixel's list
        // entry (packed position 4 B + node 4 B) and two volume bytes per
        // candidate, plus per chunk the node's 4 planes in and 4 sums out
        for (const View *v : vc)
        {
            prof->bytes += (double)v->vp->HW * (8 + 2 * P) + (double)v->vp->levelC[v->li] * (4 * 16 + 16);
            prof->pixels += (double)v->vp->HW;
        }
        prof->launches += (long)((tc.size() + MAXV - 1) / MAXV);
    }
    I.launch_edges(vc, tc, [&](auto &&go) {
        run(5, lvl_c, [&] {
            if (tp)
                prof->edges.mark(st);
            go();
            if (tp)
                prof->edges.mark(st);
        });
    });
    if (tp)
    {
        // compulsory bytes of the timed edge-message launches: per directed
        // edge its metadata (bd 8 B, bdl 4, dc 8, rev 4) and the 12 stored
        // message values read (the reverse edge's) and written; per node of
        // the level its 12 planes, 8 beliefs, RANSAC points and kept slots
        for (const View *v : vc)
        {
            const double E = v->vp->levelE[v->li], N = v->vp->levelN[v->li];
            const double bm = I.prm.msg_fp16 ? 2.0 : 4.0;
            prof->edges.bytes += E * (24.0 + 2.0 * K * bm) + N * (K * 16.0 + 2 * P * 4.0 + 16.0 + 8.0);
            prof->edges.units += E;
        }
        prof->edges.launches += (long)((tc.size() + MAXV - 1) / MAXV);
    }
    // MAP at min_level
    if (!vm.empty())
    {
        NvtxRange map_range("bp_map");
        I.launch(vm, tm, [&](const StepDesc &d) {
            run(8, vm[0]->li, [&] { k_map<<<blocks((long)d.pre[d.nt] * 32, 128), 128, 0, st>>>(nullptr, d); });
            note_launch();
        });
    }
    HBP_LAUNCH_CHECK();
    // advance every view by the action it took
    std::vector<View> keep;
    keep.reserve(I.views.size());
    for (View &v : I.views)
    {
        switch (v.phase)
        {
        case PH_INIT:
            v.phase = PH_STEP;
            v.settle();
            break;
        case PH_STEP:
        {
            const int k = v.kind();
            v.step++;
            if (k == 0)
                v.drawn.then(LcgJump(3 * P));
            if (k == 1)
                v.spatial.then(LcgJump(P));
            if (k == 2)
                v.drawn.then(LcgJump(4 * P));
            if (k == 2)
            {
                v.max_dz /= 2.0f;
                v.max_dn /= 2.0f;
            }
            if (++v.it == 6)
            {
                v.it = 0;
                ++v.i;
            }
            v.settle();
            break;
        }
        case PH_FINAL:
            if (v.li > v.vp->min_level)
            {
                if (v.vp->levels)
                    v.phase = PH_MAP_LEVEL;
                else
                    v.enter_level(v.li - 1);
            }
            else
                v.phase = PH_MAP;
            break;
        case PH_MAP_LEVEL:
            v.enter_level(v.li - 1);
            break;
        case PH_MAP:
            v.phase = PH_DONE;
            break;
        }
        if (v.phase == PH_DONE)
            finished.push_back(v.user);
        else
            keep.push_back(v);
    }
    I.views.swap(keep);
}

BpPool::BpPool(const HbpParams &prm, int streams)
{
    HbpParams quiet = prm;
    quiet.prof = nullptr; // only the first scheduler feeds the profiler
    const int S = std::max(1, std::min(streams, 64));
    try
    {
        for (int i = 0; i < S; ++i)
        {
            cudaStream_t x;
            HBP_CUDA(cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking));
            st_.push_back(x);
            sc_.push_back(std::make_unique<BpScheduler>(i == 0 ? prm : quiet, x));
        }
    }
    catch (...)
    {
        sc_.clear();
        for (cudaStream_t x : st_)
            cudaStreamDestroy(x);
        throw;
    }
}

BpPool::~BpPool()
{
    for (cudaStream_t x : st_)
        cudaStreamSynchronize(x);
    sc_.clear();
    for (cudaStream_t x : st_)
        cudaStreamDestroy(x);
}

int BpPool::pick(const ViewPlan &vp) const
{
    long windows = ceil_div(vp.HW, PC_CHUNK);
    for (auto &x : sc_)
        windows += x->windows();
    const int S = std::min(size(), bp_streams_for(windows));
    int bi = 0;
    for (int i = 1; i < S; ++i)
        if (sc_[(size_t)i]->windows() < sc_[(size_t)bi]->windows())
            bi = i;
    return bi;
}

void BpPool::add(int i, ViewPlan *vp, void *user) { sc_[(size_t)i]->add(vp, user); }

bool BpPool::active() const
{
    for (auto &x : sc_)
        if (x->active())
            return true;
    return false;
}

void BpPool::tick(std::vector<std::pair<void *, int>> &finished)
{
    std::vector<void *> fin;
    long windows = 0;
    for (auto &x : sc_)
        windows += x->windows();
    for (size_t i = 0; i < sc_.size(); ++i)
        if (sc_[i]->active())
        {
            fin.clear();
            sc_[i]->tick(fin, windows);
            for (void *f : fin)
                finished.emplace_back(f, (int)i);
        }
}

void BpPool::sync()
{
    for (cudaStream_t x : st_)
        HBP_CUDA(cudaStreamSynchronize(x));
}

// One stream below 1700 data-cost windows in flight, two below 8000, three above,
// however many views they belong to: views that fill the chip overlap on several
// streams, and small ones cost a launch each there. BP ms on 1 / 2 / 3 / 4:
//   5 x 320x240 (1500 windows) 26.5 / 27.3 / 34.2 / 44.6; 6 x 320x240 (1800)
//   28.6 / 28.0 / 34.3 / 41.3; 3 x 450x375 (1980) 31.0 / 30.3 / 37.1;
//   16 x 320x240 (4800) 53.7 / 49.9 / 52.3 / 58.1; 4 x 720x496 (5580) 67.4 / 61.5 /
//   62.2 / 66.0; 5 (6975) 81.0 / 72.6 / 74.2 / 82.0; 6 (8370) 94.1 / 85.7 / 85.2 / 89.9;
//   3 x 1080x744 (9417) 118.1 / 110.8 / 109.2; 16 x 450x375 (10560) 107.4 / 96.7 /
//   95.5 / 96.0; 16 x 720x496 (22320) 215 / 200 / 197 / 198; 4 x 1440x992 (22320)
//   260.9 / 252.9 / 249.8 / 247.5.
int bp_streams_for(long windows) { return windows < 1700 ? 1 : windows < 8000 ? 2 : 3; }

// HBP_ISP::run_ms for every view (hbp_isp.cu:1313-1346), all admitted at once,
// on a BpPool (bp_streams_for by default).
void hbp_run_views(const std::vector<ViewPlan *> &views, const HbpParams &prm, Arena &, cudaStream_t st)
{
    HBP_CUDA(cudaStreamSynchronize(st)); // the views' setup may sit on st
    long windows = 0;
    for (const ViewPlan *v : views)
        windows += ceil_div(v->HW, PC_CHUNK);
    const int S = std::min(prm.bp_streams > 0 ? prm.bp_streams : bp_streams_for(windows), (int)std::max<size_t>(views.size(), 1));
    BpPool pool(prm, S);
    for (size_t i = 0; i < views.size(); ++i)
        pool.add((int)(i % (size_t)S), views[i], views[i]);
    std::vector<std::pair<void *, int>> fin;
    while (pool.active())
        pool.tick(fin);
    pool.sync();
}

} // namespace hbp
