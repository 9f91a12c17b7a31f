// Device-wide exclusive scan and stable LSD radix sort (project kernels; the
// reference uses thrust::exclusive_scan / sort / sort_by_key at CRTrees.cu:395,
// segment.cu:1061-1064, hbp_isp.cu:888, :981, :993, :1012).
//
// A pyramid calls these some hundred times, mostly on a few thousand items, so
// what they cost is launches: a scan is one launch up to 2048 items and two
// above (no recursion), a sort one launch in all up to 8192 items, two per
// digit up to 131072 and three above.
#include "engine.h"

namespace hbp
{
namespace
{
constexpr int ST = 256, SI = 8, STILE = ST * SI; // scan tile: 2048 items

// Block-wide exclusive scan of one value per thread (T threads); returns the
// block total.
template <int T>
__device__ __forceinline__ int block_exscan(int v, int &total)
{
    __shared__ int wsum[T / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1)
    {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        wsum[w] = x;
    __syncthreads();
    if (w == 0)
    {
        int s = lane < T / 32 ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1)
        {
            int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o)
                s += y;
        }
        if (lane < T / 32)
            wsum[lane] = s;
    }
    __syncthreads();
    int base = w ? wsum[w - 1] : 0;
    total = wsum[T / 32 - 1];
    __syncthreads();
    return base + x - v;
}

// What a scan reads: an array, or 1 where a sorted edge key ends its run and
// joins two different nodes.
struct ArrayIn
{
    const int *p;
    __device__ __forceinline__ int operator()(long i) const { return p[i]; }
};
struct RunEndIn
{
    const uint64_t *keys;
    long n;
    int bits;
    __device__ __forceinline__ int operator()(long i) const { return edge_run_end(keys, n, bits, i); }
};

template <typename In>
__global__ void __launch_bounds__(ST) scan_sums(In in, long n, int *__restrict__ sums)
{
    const long t0 = (long)blockIdx.x * STILE + threadIdx.x;
    int s = 0;
#pragma unroll
    for (int k = 0; k < SI; ++k)
        s += t0 + k * ST < n ? in(t0 + k * ST) : 0;
    int total;
    block_exscan<ST>(s, total);
    if (threadIdx.x == 0)
        sums[blockIdx.x] = total;
}

// Every block adds up the sums of the tiles before its own (sums: null for a
// single tile); the last one writes the grand total.
template <typename In>
__global__ void __launch_bounds__(ST)
    scan_tiles(In in, int *__restrict__ out, long n, const int *__restrict__ sums, int *__restrict__ total_out)
{
    int before = 0, total;
    if (sums)
    {
        int s = 0;
        for (int t = threadIdx.x; t < (int)blockIdx.x; t += ST)
            s += sums[t];
        block_exscan<ST>(s, before);
    }
    const long t0 = (long)blockIdx.x * STILE + (long)threadIdx.x * SI;
    int v[SI];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SI; ++k)
    {
        v[k] = t0 + k < n ? in(t0 + k) : 0;
        s += v[k];
    }
    int ex = before + block_exscan<ST>(s, total);
#pragma unroll
    for (int k = 0; k < SI; ++k)
    {
        if (t0 + k < n)
            out[t0 + k] = ex;
        ex += v[k];
    }
    if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
        *total_out = before + total;
}

template <typename In>
void scan(In in, int *out, long n, int *total_dev, Arena &tmp, cudaStream_t st)
{
    if (n <= 0)
    {
        if (total_dev)
            HBP_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(int), st));
        return;
    }
    size_t m = tmp.mark();
    const int tiles = (int)((n + STILE - 1) / STILE);
    int *sums = nullptr;
    if (tiles > 1)
    {
        sums = tmp.alloc<int>(tiles);
        scan_sums<<<tiles, ST, 0, st>>>(in, n, sums);
        note_launch();
    }
    scan_tiles<<<tiles, ST, 0, st>>>(in, out, n, sums, total_dev);
    note_launch();
    HBP_LAUNCH_CHECK();
    tmp.rewind(m);
}

// ---------------------------------------------------------------------------
// radix sort: tiles of 2048 items processed in 8 rounds of 256 consecutive
// items; per digit the offset of (digit, tile) is the count of smaller digits
// plus that of the digit in earlier tiles, the rank inside a tile follows
// input order.
constexpr int RT = 256, RI = 8, RTILE = RT * RI;
constexpr int R_FEW = 64;     // tiles up to which a scatter block adds up the histograms itself
constexpr int RB = 1024;      // threads of the one-block sort
constexpr long R_BLOCK = 8192; // its items

template <typename KT>
__device__ __forceinline__ int digit_of(KT key, int shift)
{
    return (int)((key >> shift) & 255);
}

template <typename KT>
__global__ void __launch_bounds__(RT) radix_hist(const KT *__restrict__ keys, long n, int shift,
                                                 int *__restrict__ hist, int ntiles)
{
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const long base = (long)blockIdx.x * RTILE;
#pragma unroll
    for (int r = 0; r < RI; ++r)
    {
        long i = base + r * RT + threadIdx.x;
        if (i < n)
            atomicAdd(&h[digit_of(keys[i], shift)], 1);
    }
    __syncthreads();
    hist[(long)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Block d: digit d's counts of the tiles before each tile, in place, and its
// total.
__global__ void __launch_bounds__(ST) radix_offsets(int *__restrict__ hist, int ntiles, int *__restrict__ totals)
{
    int *row = hist + (long)blockIdx.x * ntiles;
    int before = 0, total;
    for (int t0 = 0; t0 < ntiles; t0 += ST)
    {
        const int t = t0 + threadIdx.x;
        const int v = t < ntiles ? row[t] : 0;
        const int ex = block_exscan<ST>(v, total);
        if (t < ntiles)
            row[t] = before + ex;
        before += total;
    }
    if (threadIdx.x == 0)
        totals[blockIdx.x] = before;
}

// One round of T consecutive items of a stable scatter: `run` holds where each
// digit's next item goes, `wcnt` the warps' counts.
template <typename KT, bool HAS_VAL, int T>
__device__ __forceinline__ void scatter_round(bool valid, KT key, uint32_t val, int shift, KT *okeys, uint32_t *ovals,
                                              int *run, int (*wcnt)[256])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < T / 32 * 256; i += T)
        (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const int dg = valid ? digit_of(key, shift) : 256;
    const unsigned peers = __match_any_sync(0xffffffffu, dg);
    const int wrank = __popc(peers & ((1u << lane) - 1u));
    if (valid && wrank == 0)
        wcnt[w][dg] = __popc(peers);
    __syncthreads();
    // wcnt[w][d]: counts of the warps before w; run[d] moves on by all of them
    if (threadIdx.x < 256)
    {
        int s = run[threadIdx.x];
#pragma unroll
        for (int k = 0; k < T / 32; ++k)
        {
            const int c = wcnt[k][threadIdx.x];
            wcnt[k][threadIdx.x] = s;
            s += c;
        }
        run[threadIdx.x] = s;
    }
    __syncthreads();
    if (valid)
    {
        const int pos = wcnt[w][dg] + wrank;
        okeys[pos] = key;
        if (HAS_VAL)
            ovals[pos] = val;
    }
    __syncthreads();
}

// FEW: `hist` holds the tiles' plain histograms and the block adds them up;
// otherwise the offsets and totals of radix_offsets.
template <typename KT, bool HAS_VAL, bool FEW>
__global__ void __launch_bounds__(RT)
    radix_scatter(const KT *__restrict__ keys, const uint32_t *__restrict__ vals, KT *__restrict__ okeys,
                  uint32_t *__restrict__ ovals, long n, int shift, const int *__restrict__ hist,
                  const int *__restrict__ totals, int ntiles)
{
    __shared__ int run[256];
    __shared__ int wcnt[RT / 32][256];
    const int *row = hist + (long)threadIdx.x * ntiles;
    int before = 0, all = 0, total;
    if (FEW)
        for (int t = 0; t < ntiles; ++t)
        {
            const int v = row[t];
            before += t < (int)blockIdx.x ? v : 0;
            all += v;
        }
    else
    {
        before = row[blockIdx.x];
        all = totals[threadIdx.x];
    }
    run[threadIdx.x] = before + block_exscan<RT>(all, total);
    __syncthreads();
    const long base = (long)blockIdx.x * RTILE;
    for (int r = 0; r < RI; ++r)
    {
        const long i = base + r * RT + threadIdx.x;
        const bool valid = i < n;
        scatter_round<KT, HAS_VAL, RT>(valid, valid ? keys[i] : (KT)0, HAS_VAL && valid ? vals[i] : 0u, shift, okeys,
                                       ovals, run, wcnt);
    }
}

// Every pass of a sort of up to R_BLOCK items in one block; the result lands
// in ka / va. The passes ping-pong through the alternate buffers (the block's
// own writes, ordered by its barriers).
template <typename KT, bool HAS_VAL>
__global__ void __launch_bounds__(RB) radix_block(KT *ka, uint32_t *va, KT *kb, uint32_t *vb, int n, int passes)
{
    __shared__ int run[256];
    __shared__ int wcnt[RB / 32][256];
    for (int p = 0; p < passes; ++p)
    {
        const int shift = 8 * p;
        if (threadIdx.x < 256)
            run[threadIdx.x] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += RB)
            atomicAdd(&run[digit_of(ka[i], shift)], 1);
        __syncthreads();
        int total;
        const int ex = block_exscan<RB>(threadIdx.x < 256 ? run[threadIdx.x] : 0, total);
        if (threadIdx.x < 256)
            run[threadIdx.x] = ex;
        __syncthreads();
        for (int i0 = 0; i0 < n; i0 += RB)
        {
            const int i = i0 + threadIdx.x;
            const bool valid = i < n;
            scatter_round<KT, HAS_VAL, RB>(valid, valid ? ka[i] : (KT)0, HAS_VAL && valid ? va[i] : 0u, shift, kb, vb, run,
                                           wcnt);
        }
        KT *kt = ka;
        ka = kb;
        kb = kt;
        uint32_t *vt = va;
        va = vb;
        vb = vt;
    }
    if (passes & 1) // the result lies in the alternate buffers (ka / va now), the caller's are kb / vb
        for (int i = threadIdx.x; i < n; i += RB)
        {
            kb[i] = ka[i];
            if (HAS_VAL)
                vb[i] = va[i];
        }
}

template <typename KT, bool HAS_VAL>
void radix_sort_impl(KT *keys, uint32_t *vals, KT *keys_alt, uint32_t *vals_alt, long n, int bits,
                     Arena &tmp, cudaStream_t st)
{
    if (n <= 1 || bits <= 0)
        return;
    const int passes = (bits + 7) / 8;
    if (n <= R_BLOCK)
    {
        radix_block<KT, HAS_VAL><<<1, RB, 0, st>>>(keys, vals, keys_alt, vals_alt, (int)n, passes);
        note_launch();
        HBP_LAUNCH_CHECK();
        return;
    }
    const int ntiles = (int)((n + RTILE - 1) / RTILE);
    size_t m = tmp.mark();
    int *hist = tmp.alloc<int>((size_t)256 * ntiles);
    int *totals = tmp.alloc<int>(256);
    KT *ka = keys, *kb = keys_alt;
    uint32_t *va = vals, *vb = vals_alt;
    for (int p = 0; p < passes; ++p)
    {
        int shift = 8 * p;
        radix_hist<KT><<<ntiles, RT, 0, st>>>(ka, n, shift, hist, ntiles);
        note_launch();
        if (ntiles <= R_FEW)
            radix_scatter<KT, HAS_VAL, true><<<ntiles, RT, 0, st>>>(ka, va, kb, vb, n, shift, hist, totals, ntiles);
        else
        {
            radix_offsets<<<256, ST, 0, st>>>(hist, ntiles, totals);
            note_launch();
            radix_scatter<KT, HAS_VAL, false><<<ntiles, RT, 0, st>>>(ka, va, kb, vb, n, shift, hist, totals, ntiles);
        }
        note_launch();
        HBP_LAUNCH_CHECK();
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != keys)
    {
        HBP_CUDA(cudaMemcpyAsync(keys, ka, sizeof(KT) * n, cudaMemcpyDeviceToDevice, st));
        if (HAS_VAL)
            HBP_CUDA(cudaMemcpyAsync(vals, va, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st));
    }
    tmp.rewind(m);
}
} // namespace

void exclusive_scan(const int *in, int *out, long n, int *total_dev, Arena &tmp, cudaStream_t st)
{
    scan(ArrayIn{in}, out, n, total_dev, tmp, st);
}

void scan_run_ends(const uint64_t *keys, int bits, int *out, long n, int *total_dev, Arena &tmp, cudaStream_t st)
{
    scan(RunEndIn{keys, n, bits}, out, n, total_dev, tmp, st);
}

void radix_sort_pairs_u32(uint32_t *keys, uint32_t *vals, uint32_t *keys_alt, uint32_t *vals_alt,
                          long n, int bits, Arena &tmp, cudaStream_t st)
{
    radix_sort_impl<uint32_t, true>(keys, vals, keys_alt, vals_alt, n, bits, tmp, st);
}

void radix_sort_keys_u64(uint64_t *keys, uint64_t *keys_alt, long n, int bits, Arena &tmp,
                         cudaStream_t st)
{
    radix_sort_impl<uint64_t, false>(keys, nullptr, keys_alt, nullptr, n, bits, tmp, st);
}

} // namespace hbp
