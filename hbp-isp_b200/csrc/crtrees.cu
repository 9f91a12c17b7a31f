// CRTrees: connected components of a directed 1-NN (functional) graph.
//
// Reference: CRTrees::get_clus (CRTrees.cu:315-354) with compute_in_degree,
// check_larger_than_one, de_link_and_compute_mask, one_step_jump, re_link,
// re_link_all, one_step_jump_max (:28-187, driven by :207-312) and
// compact_clus_label (:357-403).
// The reference drives every pointer-jumping step from the host and reads a
// flag back after each; here the whole procedure is one kernel. Its phases are
// separated by bounded grid barriers (a cooperative launch), or, for graphs of
// up to CRT_SMEM_NODES nodes, by block barriers: one block then holds every
// array in shared memory and also ranks the labels, which costs one launch in
// all. Each phase reads the state left by the previous one (re_link reads a
// snapshot), which is the race-free reading of the reference's kernels; the
// labels it produces are those of the reference (checked against the
// reference build on random graphs and on every pyramid level).
#include <mutex>

#include "engine.h"

namespace hbp
{
namespace
{
constexpr int CR_T = 512; // 256: 1.64 ms for the superpixels of a 720x496 image, 512: 1.53, 1024: 1.52
constexpr int MAX_ROUNDS = 48, MAX_JUMPS = 64, MAX_FLAGS = MAX_ROUNDS * (MAX_JUMPS + 2) + MAX_JUMPS + 8;

// The arrays of a run. M and Kb (the label phase) may share indeg's and old's
// memory.
struct CrBufs
{
    int *C, *Nb, *nn, *indeg, *M, *Kb;
    uint8_t *mask, *maskc;
};

// How the phases of a run meet: every thread of the grid, or of one block.
// vote(any) ends a phase: false if the wait gave up, `any` then true if any
// thread passed true.
struct GridPhases
{
    int *flags;
    GridBarrier bar;
    int ph = 0; // flags used so far
    __device__ __forceinline__ int first() const { return blockIdx.x * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ int stride() const { return gridDim.x * blockDim.x; }
    __device__ __forceinline__ bool sync() { return grid_sync(bar, gridDim.x); }
    __device__ __forceinline__ bool full() const { return ph + MAX_JUMPS + 2 >= MAX_FLAGS; }
    __device__ __forceinline__ bool vote(bool &any)
    {
        const int f = ph++;
        if (__syncthreads_or(any) && threadIdx.x == 0)
            atomicOr(&flags[f], 1);
        if (!sync())
            return false;
        any = *(volatile int *)&flags[f] != 0;
        return true;
    }
};
struct BlockPhases
{
    __device__ __forceinline__ int first() const { return threadIdx.x; }
    __device__ __forceinline__ int stride() const { return blockDim.x; }
    __device__ __forceinline__ bool sync()
    {
        __syncthreads();
        return true;
    }
    __device__ __forceinline__ bool full() const { return false; }
    __device__ __forceinline__ bool vote(bool &any)
    {
        any = __syncthreads_or(any);
        return true;
    }
};

// Runs CRTrees on the successors b.nn (C = nn, mask = 1, indeg = 0 on entry);
// the labels end in the returned array (b.M or b.Kb). Null: a wait timed out,
// or no convergence (recorded in err).
template <typename Phases>
__device__ __forceinline__ int *crtrees_run(int N, CrBufs b, Phases &p, int *err)
{
    const int t0 = p.first(), stride = p.stride();
    int *C = b.C, *Nb = b.Nb, *nn = b.nn, *indeg = b.indeg;
    uint8_t *mask = b.mask, *maskc = b.maskc;
    for (int round = 0;; ++round)
    {
        if (round >= MAX_ROUNDS || p.full())
        {
            if (t0 == 0)
                atomicExch(err, (int)DERR_NO_CONVERGENCE);
            return nullptr;
        }
        // compute_in_degree and check_larger_than_one: does an active node get
        // a second active predecessor?
        bool any = false;
        for (int i = t0; i < N; i += stride)
            if (mask[i])
            {
                const int c = C[i];
                if (atomicAdd(&indeg[c], 1) >= 1 && mask[c])
                    any = true;
            }
        if (!p.vote(any))
            return nullptr;
        if (!any)
            break;
        // de_link_and_compute_mask
        for (int i = t0; i < N; i += stride)
        {
            const int m = indeg[i] > 1;
            maskc[i] = mask[i];
            mask[i] = (uint8_t)m;
            if (m)
                C[i] = i;
        }
        if (!p.sync())
            return nullptr;
        // pointer_jumping: odd steps write Nb from C, even steps C from Nb
        int *cur = C, *oth = Nb;
        for (int j = 0;; ++j)
        {
            if (j >= MAX_JUMPS)
            {
                if (t0 == 0)
                    atomicExch(err, (int)DERR_NO_CONVERGENCE);
                return nullptr;
            }
            any = false;
            for (int i = t0; i < N; i += stride)
                if (maskc[i])
                {
                    int a = cur[i], c2 = cur[a];
                    oth[i] = c2;
                    if (!mask[a] && mask[c2])
                        any = true;
                }
            if (!p.vote(any))
                return nullptr;
            int *t = cur;
            cur = oth;
            oth = t;
            if (!any)
                break;
        }
        // re_link: from buffer C after jumping (a snapshot: it writes Nb)
        for (int i = t0; i < N; i += stride)
        {
            int v = C[i];
            if (mask[i])
            {
                const int s = nn[i];
                v = mask[s] ? s : C[s];
            }
            else if (!maskc[i] && maskc[v])
                v = C[v];
            Nb[i] = v;
        }
        if (!p.sync())
            return nullptr;
        // re_link_all; its result is the next round's C
        for (int i = t0; i < N; i += stride)
        {
            const int v = Nb[i];
            int s = nn[i];
            if (mask[i])
                s = v;
            else if (mask[v])
                s = Nb[v];
            nn[i] = s;
            C[i] = s;
            indeg[i] = 0;
        }
        if (!p.sync())
            return nullptr;
    }
    // pointer_jumping_max: label = max node index along the successor chain
    int *cn = C, *on = Nb, *cm = b.M, *om = b.Kb;
    for (int i = t0; i < N; i += stride)
        cm[i] = C[i];
    if (!p.sync())
        return nullptr;
    for (int j = 0;; ++j)
    {
        if (j >= MAX_JUMPS)
        {
            if (t0 == 0)
                atomicExch(err, (int)DERR_NO_CONVERGENCE);
            return nullptr;
        }
        bool any = false;
        for (int i = t0; i < N; i += stride)
        {
            int a = cn[i];
            int m = max(cm[i], cm[a]);
            om[i] = m;
            on[i] = cn[a];
            if (m != cm[i])
                any = true;
        }
        if (!p.vote(any))
            return nullptr;
        int *t = cn;
        cn = on;
        on = t;
        t = cm;
        cm = om;
        om = t;
        if (!any)
            return cm;
    }
}

// label[i], and used[l] = 1 for every label l.
__global__ void __launch_bounds__(CR_T)
    crtrees_kernel(const int *__restrict__ nn_in, int N, CrBufs b, int *__restrict__ label, int *__restrict__ used,
                   int *flags, GridBarrier bar, int *err)
{
    GridPhases p{flags, bar};
    for (int i = p.first(); i < N; i += p.stride())
    {
        const int v = nn_in[i];
        b.nn[i] = v;
        b.C[i] = v;
        b.mask[i] = 1;
        b.indeg[i] = 0;
        used[i] = 0;
    }
    if (!p.sync())
        return;
    const int *l = crtrees_run(N, b, p, err);
    if (!l)
        return;
    for (int i = p.first(); i < N; i += p.stride())
    {
        label[i] = l[i];
        used[l[i]] = 1;
    }
}

__global__ void remap_labels(const int *label, const int *pos, int N, int *clus)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N)
    {
        // a kernel that gave up (error word set) may leave garbage
        int l = label[i];
        clus[i] = (l >= 0 && l < N) ? pos[l] : 0;
    }
}

// The whole procedure for small graphs in one block: every array in shared
// memory (22 bytes a node), the labels ranked by the block. A grid barrier
// costs 1 - 2 us and a run has some sixty phases: the pyramid's small levels took
// 150 - 185 us each with 2 - 22 blocks and five more launches.
constexpr int CRT_BT = 1024;
constexpr int CRT_SMEM_NODES = 10000;
constexpr size_t crt_smem(int N) { return (size_t)N * 22 + 64; }

__global__ void __launch_bounds__(CRT_BT) crtrees_block(const int *__restrict__ nn_in, int N, int *__restrict__ clus,
                                                        int *num, int *err)
{
    extern __shared__ int crt_sm[];
    __shared__ int wsum[CRT_BT / 32];
    CrBufs b;
    b.C = crt_sm;
    b.Nb = b.C + N;
    b.nn = b.Nb + N;
    b.indeg = b.nn + N;
    b.M = b.indeg; // the in-degrees are done with before the labels start
    b.Kb = b.indeg + N;
    b.mask = reinterpret_cast<uint8_t *>(b.Kb + N);
    b.maskc = b.mask + N;
    BlockPhases p;
    for (int i = threadIdx.x; i < N; i += CRT_BT)
    {
        const int v = nn_in[i];
        b.nn[i] = v;
        b.C[i] = v;
        b.mask[i] = 1;
        b.indeg[i] = 0;
    }
    __syncthreads();
    const int *l = crtrees_run(N, b, p, err);
    if (!l) // block-uniform
    {
        for (int i = threadIdx.x; i < N; i += CRT_BT)
            clus[i] = 0;
        if (threadIdx.x == 0)
            *num = 0;
        return;
    }
    // compact_clus_label: rank labels in increasing order, a run of nodes per
    // thread (nn: used flags, then ranks)
    int *used = b.nn;
    for (int i = threadIdx.x; i < N; i += CRT_BT)
        used[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += CRT_BT)
        used[l[i]] = 1;
    __syncthreads();
    const int per = (N + CRT_BT - 1) / CRT_BT, i0 = min((int)threadIdx.x * per, N), i1 = min(i0 + per, N);
    int s = 0;
    for (int i = i0; i < i1; ++i)
        s += used[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = s;
    for (int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        wsum[w] = x;
    __syncthreads();
    int before = x - s, total = 0;
    for (int k = 0; k < CRT_BT / 32; ++k)
    {
        before += k < w ? wsum[k] : 0;
        total += wsum[k];
    }
    for (int i = i0; i < i1; ++i)
    {
        const int u = used[i];
        used[i] = before;
        before += u;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += CRT_BT)
        clus[i] = used[l[i]];
    if (threadIdx.x == 0)
        *num = total;
}

// Grid size of the cooperative CRTrees launch on the current device: one
// block per SM at most, which leaves room for concurrent lanes (each lane may
// run its own cooperative CRTrees launch). Computed once per device; lanes on
// several host threads may ask at the same time.
int coop_blocks(int N)
{
    static std::mutex mu;
    static int max_blocks[64] = {};
    int dev;
    HBP_CUDA(cudaGetDevice(&dev));
    int mb;
    {
        std::lock_guard<std::mutex> lk(mu);
        mb = dev >= 0 && dev < 64 ? max_blocks[dev] : 0;
    }
    if (!mb)
    {
        int sms, per_sm = 0;
        HBP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        HBP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, crtrees_kernel, CR_T, 0));
        mb = sms * (per_sm > 1 ? 1 : per_sm);
        if (mb < 1)
            mb = 1;
        std::lock_guard<std::mutex> lk(mu);
        if (dev >= 0 && dev < 64)
            max_blocks[dev] = mb;
    }
    int want = ceil_div(N, CR_T * 4);
    return want < 1 ? 1 : (want > mb ? mb : want);
}

// crtrees_block's shared memory exceeds the default limit; the attribute is
// set once per device.
void allow_block_smem()
{
    static std::mutex mu;
    static bool done[64] = {};
    int dev;
    HBP_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 64 && done[dev])
        return;
    HBP_CUDA(cudaFuncSetAttribute(crtrees_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)crt_smem(CRT_SMEM_NODES)));
    if (dev >= 0 && dev < 64)
        done[dev] = true;
}
} // namespace

void crtrees_labels(const int *nn, int N, int *clus, int *num_dev, int *err_dev, Arena &tmp,
                    cudaStream_t st)
{
    if (N <= CRT_SMEM_NODES)
    {
        allow_block_smem();
        crtrees_block<<<1, CRT_BT, crt_smem(N), st>>>(nn, N, clus, num_dev, err_dev);
        note_launch();
        HBP_LAUNCH_CHECK();
        return;
    }
    size_t m = tmp.mark();
    CrBufs b;
    b.C = tmp.alloc<int>(N);
    b.Nb = tmp.alloc<int>(N);
    b.nn = tmp.alloc<int>(N);
    b.indeg = tmp.alloc<int>(N);
    b.M = tmp.alloc<int>(N);
    b.Kb = tmp.alloc<int>(N);
    b.mask = tmp.alloc<uint8_t>(N);
    b.maskc = tmp.alloc<uint8_t>(N);
    int *label = tmp.alloc<int>(N), *used = tmp.alloc<int>(N);
    int *flags = tmp.alloc<int>(MAX_FLAGS + 1); // and the barrier's counter
    HBP_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * (MAX_FLAGS + 1), st));
    GridBarrier gb{reinterpret_cast<unsigned int *>(flags + MAX_FLAGS), err_dev};
    int nb = coop_blocks(N);
    void *args[] = {(void *)&nn, (void *)&N, (void *)&b, (void *)&label, (void *)&used, (void *)&flags, (void *)&gb,
                    (void *)&err_dev};
    HBP_CUDA(cudaLaunchCooperativeKernel((const void *)crtrees_kernel, dim3(nb), dim3(CR_T), args, 0, st));
    note_launch();
    // compact_clus_label: rank labels in increasing order
    int *pos = b.Nb; // reuse
    exclusive_scan(used, pos, N, num_dev, tmp, st);
    remap_labels<<<ceil_div(N, 256), 256, 0, st>>>(label, pos, N, clus);
    note_launch();
    HBP_LAUNCH_CHECK();
    tmp.rewind(m);
}

// A bounded wait that nothing ends: one block waits at a grid barrier for a
// second block that is never launched; after spin_limit polls the barrier
// records DERR_BARRIER_TIMEOUT and the kernel returns (the check that a
// device wait ends with a status instead of hanging).
__global__ void barrier_probe_kernel(GridBarrier bar, long spin_limit) { grid_sync(bar, 2u, spin_limit); }

void launch_barrier_probe(unsigned int *count, int *err, long spin_limit, cudaStream_t st)
{
    GridBarrier b{count, err};
    barrier_probe_kernel<<<1, 32, 0, st>>>(b, spin_limit);
    note_launch();
    HBP_LAUNCH_CHECK();
}

} // namespace hbp
