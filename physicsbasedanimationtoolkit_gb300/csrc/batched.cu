// The persistent batched step (see batched.cuh for the work items and the progress argument).
#include "batched.cuh"
#include "sweep_device.cuh"

#include <climits>

namespace pbgb {

namespace {

__device__ __forceinline__ int32_t load_acquire(int32_t const* q)
{
    int32_t v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(q) : "memory");
    return v;
}

__device__ __forceinline__ void add_release(int32_t* q, int32_t v)
{
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(q), "r"(v) : "memory");
}

__device__ __forceinline__ void copy_async(int4* to, int4 const* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(to))), "l"(from) : "memory");
}

__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits until *counter >= need.  Returns false when the wait gave up (time limit, or another
// block's wait gave up before): then flags[1] and the abort flag are set.  At most 2^24 polls in
// any case, so the loop ends even if the timer stood still.
__device__ bool wait_for(BatchedStepParams const& p, int32_t const* counter, int32_t need)
{
    if (load_acquire(counter) >= need)
        return true;
    unsigned long long const t0 = global_ns();
    unsigned sleep              = 32;
    for (int poll = 0; poll < (1 << 24); ++poll)
    {
        if (load_acquire(counter) >= need)
            return true;
        if (*reinterpret_cast<int32_t const volatile*>(p.words + kBatchWordStride) != 0)
            return false;
        if (static_cast<long long>(global_ns() - t0) > p.waitNs)
            break;
        __nanosleep(sleep);
        sleep = sleep < 1024 ? 2 * sleep : sleep;
    }
    atomicOr(p.flags + 1, 1);
    atomicExch(p.words + kBatchWordStride, 1);
    return false;
}

// Bound by memory: DRAM for batches larger than L2 (20 B per pair of incidences, 8 B per neighbour, the
// positions that leave L2 between two colours of a mesh).  64 cubes of 6^3 to 32^3, 20 iterations: 3.05
// ms with 24 B per incidence, 2.75 ms with 12 B, 2.37 ms with pairs and 2 lanes, 2.28 ms with four
// neighbours in flight per lane and 4 lanes, 2.26 ms with the counters on lines of their own, 2.08 ms
// with blocks of 64, 2.06 ms with the table of one iteration (its first step 3.2 ms, 11.5 ms before).
//
// Colour sweep of solve entries [begin, end) by the whole block: sub-tiles of blockDim / L vertices,
// each staged and solved like staged_sweep_kernel (the same arithmetic in the same order), with the
// block's positions read through L2.  The pair loop keeps two pairs' records in flight
// (this one's and the next two's loads overlap its arithmetic): the batch's records
// stream from DRAM, and one record ahead per lane left too few bytes in flight per SM.  (Loading
// the records evict-first, ld.global.cs, doubled the DRAM reads of a 256-mesh step: a record's
// sector left L2 before the neighbouring lanes had read their parts of it.)
template <int L, bool CHEB>
__device__ __forceinline__ void sweep_tile(BatchedStepParams const& bp, SweepParams const& p, int32_t const volatile* iteration, int begin, int end, float4* slab)
{
    constexpr int kNbrs = L >= 16 ? 1 : (L >= 8 ? 2 : 4);
    int const per  = int(blockDim.x) / L;
    int const lane = int(threadIdx.x) & (L - 1);
    for (int f = begin; f < end; f += per)
    {
        int const s      = f + int(threadIdx.x) / L;
        bool const valid = s < end;
        int const nb0    = __ldg(p.nbrPtr + f);
        VertexBlock<float> b;
        zero(b);
        int i       = 0;
        float xi[3] = {0.f, 0.f, 0.f};
        int k = 0, k1 = 0, n0 = 0, n1 = 0, base = 0;
        uint32_t q0 = 0u, q1 = 0u;
        float4 mt0 = make_float4(0.f, 0.f, 0.f, 0.f), mt1 = mt0;
        if (valid)
        {
            i    = __ldg(p.solve + s);
            n0   = __ldg(p.nbrPtr + s);
            n1   = __ldg(p.nbrPtr + s + 1);
            base = n0 - nb0;
            k1   = __ldg(p.pairPtr + s + 1);
            k    = __ldg(p.pairPtr + s) + lane;
            if (k < k1)
            {
                q0  = __ldg(p.pairSlots + k);
                mt0 = __ldg(p.pairMat + k);
            }
            if (k + L < k1)
            {
                q1  = __ldg(p.pairSlots + k + L);
                mt1 = __ldg(p.pairMat + k + L);
            }
            load3(Mem<true>::ld((CHEB ? p.hprev : p.x) + i), xi);
            // kNbrs neighbours' records, then their positions, in flight together.
            for (int j = n0 + lane; j < n1; j += kNbrs * L)
            {
                uint2 a[kNbrs];
                float4 xa[kNbrs];
#pragma unroll
                for (int u = 0; u < kNbrs; ++u)
                    a[u] = __ldg(p.nbr + min(j + u * L, n1 - 1));
#pragma unroll
                for (int u = 0; u < kNbrs; ++u)
                    xa[u] = Mem<true>::ld((CHEB && !(a[u].x >> 31) ? p.hprev : p.x) + (a[u].x & kIndexMask));
#pragma unroll
                for (int u = 0; u < kNbrs; ++u)
                    if (j + u * L < n1)
                        stage_neighbour(b, slab + base + j + u * L - n0, xa[u], xi, __uint_as_float(a[u].y));
            }
        }
        __syncwarp();
        if (valid)
        {
            for (; k < k1; k += L)
            {
                uint32_t q2 = 0u;
                float4 mt2  = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k + 2 * L < k1)
                {
                    q2  = __ldg(p.pairSlots + k + 2 * L);
                    mt2 = __ldg(p.pairMat + k + 2 * L);
                }
                staged_pair(b, slab + base, q0, mt0);
                q0  = q1;
                mt0 = mt1;
                q1  = q2;
                mt1 = mt2;
            }
        }
        if constexpr (CHEB)
        {
            // Read now: held over the loops, they would not fit the registers.
            SweepParams q = p;
            q.k           = *iteration;
            q.omega       = __ldg(bp.omega + q.k);
            q.hcur        = q.k & 1 ? bp.H1 : bp.H0;
            finish_vertex<L, CHEB, false, false, true>(q, b, valid, lane, i, s, xi);
        }
        else
            finish_vertex<L, CHEB, false, false, true>(p, b, valid, lane, i, s, xi);
        if (f + per < end)
            __syncthreads(); // the next sub-tile reuses the slab
    }
}

template <int L, bool CHEB>
__global__ void __launch_bounds__(256, 4) batched_step_kernel(BatchedStepParams p)
{
    extern __shared__ float4 slab[];
    // Words of the item to run and (filled at its end) of the one after it: x = -1, no items left; y = -1, the
    // wait gave up.
    __shared__ int4 sItem[2], sNeed[2];
    __shared__ int32_t sIter[2];
    // Group of the last ticket (thread 0): its first ticket, iteration (-1: begin items, iterations: end
    // items) and substep; poison: substep -1 in sSub.
    __shared__ int32_t sBase, sGroup, sSubstep, sSub;
    int32_t next = 0;
    auto fetch   = [&](int32_t it, int slot) {
        if (it >= p.nItems)
        {
            sItem[slot].x = -1;
            return;
        }
        // Tickets only grow: step from group to group (two integer divisions took 0.2 us an item).
        int32_t base = sBase, k = sGroup, s = sSubstep, at = 0;
        for (;;)
        {
            int32_t const n = k < 0 ? p.nBegin : (k < p.iterations ? p.nSweep : p.nEnd);
            if (it - base < n)
                break;
            base += n;
            if (k == p.iterations)
            {
                k = -1;
                ++s;
            }
            else
                ++k;
        }
        at = it - base + (k < 0 ? 0 : (k < p.iterations ? p.nBegin : p.nBegin + p.nSweep));
        copy_async(&sItem[slot], &p.items[at].a);
        copy_async(&sNeed[slot], &p.items[at].b);
        sBase       = base;
        sGroup      = k;
        sSubstep    = s;
        sSub        = it == p.poison ? -1 : s;
        sIter[slot] = max(k, 0);
    };
    if (threadIdx.x == 0)
    {
        sBase = sSubstep = 0;
        sGroup           = -1;
        fetch(atomicAdd(p.words, 1), 0);
    }
    for (int slot = 0;; slot ^= 1)
    {
        if (threadIdx.x == 0)
        {
            copy_async_wait();
            int32_t const mesh = sItem[slot].x;
            if (mesh >= 0)
            {
                int4 const n       = sNeed[slot];
                int32_t const need = sSub < 0 ? INT_MAX : n.x + sIter[slot] * n.y + sSub * n.z;
                next               = atomicAdd(p.words, 1); // taken now, used after this item
                if (!wait_for(p, p.words + (2 + mesh) * kBatchWordStride, need))
                    sItem[slot].y = -1;
            }
        }
        __syncthreads();
        int4 const a = sItem[slot];
        if (a.x < 0)
            break;
        if (a.y >= 0)
        {
            int const kind = a.y;
            if (kind == kBatchSweep)
            {
                SweepParams q = p.sweep;
                if constexpr (CHEB)
                    q.hprev = (sIter[slot] + 1) & 1 ? p.H1 : p.H0;
                sweep_tile<L, CHEB>(p, q, &sIter[slot], a.z, a.w, slab);
            }
            else if (kind == kBatchBegin)
            {
                for (int v = a.z + int(threadIdx.x); v < a.w; v += int(blockDim.x))
                    begin_substep_vertex<true>(p.sub, v);
            }
            else
            {
                for (int v = a.z + int(threadIdx.x); v < a.w; v += int(blockDim.x))
                    end_substep_vertex<true>(p.sub, v);
            }
        }
        // The next item's words load while the block's other warps finish this one.
        if (threadIdx.x == 0)
            fetch(next, slot ^ 1);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            __threadfence();
            add_release(p.words + (2 + sItem[slot].x) * kBatchWordStride, 1);
        }
    }
}

template <int L, bool CHEB>
cudaError_t launch_l(BatchedStepParams const& p, int block, int grid, size_t smem, cudaStream_t s)
{
    batched_step_kernel<L, CHEB><<<grid, block, smem, s>>>(p);
    return cudaGetLastError();
}

template <bool CHEB>
cudaError_t launch_c(BatchedStepParams const& p, int lanes, int block, int grid, size_t smem, cudaStream_t s)
{
    switch (lanes)
    {
        case 1: return launch_l<1, CHEB>(p, block, grid, smem, s);
        case 2: return launch_l<2, CHEB>(p, block, grid, smem, s);
        case 4: return launch_l<4, CHEB>(p, block, grid, smem, s);
        case 8: return launch_l<8, CHEB>(p, block, grid, smem, s);
        case 16: return launch_l<16, CHEB>(p, block, grid, smem, s);
        case 32: return launch_l<32, CHEB>(p, block, grid, smem, s);
        default: return cudaErrorInvalidValue;
    }
}

template <bool CHEB>
void const* kernel_of(int lanes)
{
    switch (lanes)
    {
        case 1: return reinterpret_cast<void const*>(batched_step_kernel<1, CHEB>);
        case 2: return reinterpret_cast<void const*>(batched_step_kernel<2, CHEB>);
        case 4: return reinterpret_cast<void const*>(batched_step_kernel<4, CHEB>);
        case 8: return reinterpret_cast<void const*>(batched_step_kernel<8, CHEB>);
        case 16: return reinterpret_cast<void const*>(batched_step_kernel<16, CHEB>);
        case 32: return reinterpret_cast<void const*>(batched_step_kernel<32, CHEB>);
        default: return nullptr;
    }
}

} // namespace

cudaError_t launch_batched_step(BatchedStepParams const& p, int lanes, int block, int grid, size_t smem, bool chebyshev, cudaStream_t s)
{
    if (p.nItems <= 0)
        return cudaSuccess;
    if (grid < 1 || block < 32 || block > 256 || block % lanes != 0 || smem > kStagedMaxBytes || !p.items ||
        !p.words || !p.flags || !p.sweep.pairMat || !p.sweep.pairSlots || !p.sweep.nbrPtr || (chebyshev && (!p.H0 || !p.H1 || !p.omega)))
        return cudaErrorInvalidValue;
    return chebyshev ? launch_c<true>(p, lanes, block, grid, smem, s) : launch_c<false>(p, lanes, block, grid, smem, s);
}

int batched_step_blocks_per_sm(int lanes, int block, size_t smem, bool chebyshev)
{
    void const* k = chebyshev ? kernel_of<true>(lanes) : kernel_of<false>(lanes);
    if (!k)
        return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, block, smem) != cudaSuccess)
    {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t prepare_batched_step()
{
    int const lanes[] = {1, 2, 4, 8, 16, 32};
    for (bool cheb : {false, true})
        for (int L : lanes)
        {
            void const* k = cheb ? kernel_of<true>(L) : kernel_of<false>(L);
            cudaError_t const e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kStagedMaxBytes));
            if (e != cudaSuccess)
                return e;
        }
    return cudaSuccess;
}

} // namespace pbgb
