// The cluster step (see cluster_step.cuh).
#include "cluster_step.cuh"
#include "sweep_device.cuh"

namespace pbgb {

namespace {

// All threads of the cluster (of the block, for a cluster of one).  Orders shared and global memory.
template <bool CLUSTER>
__device__ __forceinline__ void cluster_sync()
{
    if constexpr (CLUSTER)
    {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    else
        __syncthreads();
}

__device__ __forceinline__ uint32_t shared_address(void const* q)
{
    return uint32_t(__cvta_generic_to_shared(q));
}

__device__ __forceinline__ uint32_t remote_address(uint32_t local, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}

// Stores v at the remote shared address `to` and adds its 16 bytes to the remote barrier `bar`.
__device__ __forceinline__ void store_async(uint32_t to, uint32_t bar, float4 v)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void barrier_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_address(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void barrier_expect(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void barrier_arrive(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(count) : "memory");
}

// Whether the barrier's phase `parity` is over (suspends the thread for a while when not).  CLUSTER: what
// other blocks stored with the phase's bytes is then visible (an acquire at the block's scope orders the
// block's own copies only).
template <bool CLUSTER>
__device__ __forceinline__ bool barrier_passed(uint32_t a, uint32_t parity)
{
    uint32_t done;
    if constexpr (CLUSTER)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
    else
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
    return done != 0u;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the end of the barrier's phase `parity`; false when it gave up: after `ns` nanoseconds, or at
// once when another wait of the block (gaveUp) or of the launch (flags[1], which the host reports) has.
template <bool CLUSTER>
__device__ __noinline__ bool barrier_wait_slow(uint32_t a, uint32_t parity, int32_t volatile* gaveUp, int32_t* flags, long long ns)
{
    unsigned long long const t0 = global_ns();
    for (;;)
    {
        if (barrier_passed<CLUSTER>(a, parity))
            return true;
        if (*gaveUp || *reinterpret_cast<int32_t const volatile*>(flags + 1) ||
            static_cast<long long>(global_ns() - t0) > ns)
            break;
    }
    *gaveUp = 1;
    atomicOr(flags + 1, 1);
    return false;
}

template <bool CLUSTER = false>
__device__ __forceinline__ bool barrier_wait(uint64_t* bar, uint32_t parity, int32_t volatile* gaveUp, int32_t* flags, long long ns)
{
    uint32_t const a = shared_address(bar);
    return barrier_passed<CLUSTER>(a, parity) || barrier_wait_slow<CLUSTER>(a, parity, gaveUp, flags, ns);
}

// When a wait gives up, the tile that did not arrive is never read and a barrier whose phase did not end is
// not arrived on again; the warps run down the step's block and cluster barriers.  The positions are then
// not valid, which the host reports.
//
// Registers: two blocks share an SM at 80 and often do not at 88, and clusters of 16 blocks find room in few
// places: 9 meshes of 4^3 to 12^3 take 65 us a step at 80 and 94 at 87 (two rounds of clusters).  None of the
// limits spills.  Streamed tiles and two-buffer sums lose more than that gains below 96 (a 5,040-vertex
// Chebyshev step 124 us at 96, 127 at 88, 129 at 80), so those lanes that large parts take keep 96.
template <int L, bool CHEB, bool REC, bool CLUSTER>
constexpr int kClusterRegisters = REC ? 96 : (!CLUSTER || (!CHEB && (L == 1 || L >= 8)) ? 80 : (CHEB && (L == 1 || L == 32) ? 88 : 96));

template <int L, bool CHEB, bool REC, bool CLUSTER>
__global__ void __maxnreg__((kClusterRegisters<L, CHEB, REC, CLUSTER>)) cluster_step_kernel(ClusterStepParams p)
{
    // Neighbours a lane has in flight at once: a block holds few warps, so a lane's own independent
    // loads hide the latency of shared memory.
    constexpr int kNbrs = L >= 16 ? 1 : (L >= 8 ? 2 : 4);
    extern __shared__ __align__(128) unsigned char shared[];
    __shared__ int32_t sGaveUp;
    int32_t volatile* const gaveUp = &sGaveUp;
    // Ring stages, barriers, positions, slabs.
    unsigned char* const ring = shared;
    uint64_t* const full  = reinterpret_cast<uint64_t*>(ring + size_t(p.stages) * size_t(p.stageBytes));
    uint64_t* const empty = full + p.stages;
    uint64_t* const halo  = empty + p.stages;
    int2* const color     = reinterpret_cast<int2*>(halo + p.nColors); // the part's partColor
    float4* const T       = reinterpret_cast<float4*>(color + p.nColors); // own: inertial target, m / h^2
    float4* const X       = T + p.ownedCapacity;                          // raw positions
    float4* const A       = CHEB ? X + p.localCapacity : X;               // accelerated iterates
    float4* const B       = A + p.localCapacity;                          // Chebyshev: own, one iterate back
    int const warp        = int(threadIdx.x >> 5);
    int const warps       = int(blockDim.x >> 5) - 1; // solving warps; the last one streams the tiles
    int const wlane       = int(threadIdx.x & 31);
    int const part        = int(blockIdx.x);
    int const tile0       = __ldg(p.partTile + part);
    int const nTiles      = __ldg(p.partTile + part + 1) - tile0;
    bool const resident   = nTiles <= p.stages;
    SubstepParams const& sub = p.sub;
    int32_t* const flags     = sub.flags;
    long long const ns       = p.waitNs;

    if (threadIdx.x == 0)
    {
        sGaveUp = 0;
        for (int i = 0; i < p.stages; ++i)
        {
            barrier_init(full + i, 1);
            barrier_init(empty + i, L);
        }
        for (int c = 0; c < p.nColors; ++c)
        {
            barrier_init(halo + c, 1);
            color[c] = __ldg(p.partColor + size_t(part) * size_t(p.nColors) + size_t(c));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    if (warp == warps)
    {
        // The producer: every tile of every iteration in order (once, when all stay).
        int stage = 0, issued = 0;
        uint32_t round = 0;
        bool issuing   = wlane == 0;
        int const poison = blockIdx.x == 0 ? p.poison : -1; // a tile that never comes (tests)
        for (int ss = 0; ss < p.substeps; ++ss)
        {
            cluster_sync<CLUSTER>();
            if (issuing && (!resident || ss == 0))
            {
                int const passes = resident ? (p.iterations > 0 ? 1 : 0) : p.iterations;
                for (int k = 0; k < passes && issuing; ++k)
                    for (int t = 0; t < nTiles; ++t)
                    {
                        if (round > 0 && !barrier_wait(empty + stage, (round - 1) & 1u, gaveUp, flags, ns))
                        {
                            issuing = false;
                            break;
                        }
                        int2 const d = __ldg(p.tiles + tile0 + t);
                        barrier_expect(full + stage, uint32_t(d.y));
                        if (issued != poison)
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                             shared_address(ring + size_t(stage) * size_t(p.stageBytes))),
                                         "l"(p.tileData + size_t(d.x) * 16), "r"(d.y), "r"(shared_address(full + stage))
                                         : "memory");
                        ++issued;
                        if (++stage == p.stages)
                        {
                            stage = 0;
                            ++round;
                        }
                    }
            }
            __syncwarp();
            if (ss + 1 == p.substeps && wlane == 0)
            {
                // No copy is on its way when the block ends, also when a wait gave up.
                unsigned long long const t0 = global_ns();
                for (int i = max(issued - p.stages, 0); i < issued; ++i)
                    while (i != poison && !barrier_passed<false>(shared_address(full + i % p.stages), uint32_t(i / p.stages) & 1u) &&
                           static_cast<long long>(global_ns() - t0) <= ns)
                        ;
            }
            __syncwarp();
            if (CLUSTER || ss + 1 < p.substeps)
                cluster_sync<CLUSTER>();
        }
        return;
    }

    int const v0      = __ldg(p.partPtr + part);
    int const nLocal  = __ldg(p.partPtr + part + 1) - v0;
    int const nOwned  = __ldg(p.partOwned + part);
    int const threads = 32 * warps;
    int const lane    = int(threadIdx.x) & (L - 1);
    float4* const slabs     = CHEB ? B + p.ownedCapacity : B;
    float4* const slab      = slabs + warp * p.slabPerWarp;
    float4* const XT        = slabs + warps * p.slabPerWarp; // own, with damping: the substep's start
    int stage0 = 0;       // stage of the colour's first tile
    uint32_t round0 = 0u; // times the ring came round before it
    bool solving    = true; // the warp's (no wait gave up)

    for (int ss = 0; ss < p.substeps; ++ss)
    {
        size_t const n = size_t(sub.n);
        float4 *tapeX = nullptr, *tapeRaw = nullptr, *tapeH = nullptr;
        if constexpr (REC)
        {
            tapeX   = p.tapeX + size_t(ss) * size_t(p.tapeIterations + 1) * n;
            tapeH   = p.tapeH + size_t(ss) * size_t(p.tapeIterations) * size_t(p.nFree) * 2;
            tapeRaw = CHEB ? p.tapeRaw + size_t(ss) * size_t(p.tapeIterations) * n : nullptr;
        }
        // Inertial target and initial guess.  A block forms the guesses of its halo itself; the own
        // vertices' x in global memory is written at the end of the substep only, after every block
        // has read it here.
        for (int j = int(threadIdx.x); j < nLocal; j += threads)
        {
            uint32_t const word = __ldg(p.partVertex + v0 + j);
            int const i         = int(word & kIndexMask);
            bool const own      = j < nOwned;
            float4 const x4     = __ldcg(sub.x + i);
            if (REC && own)
            {
                float4* const start = p.tapeS + size_t(ss) * 3 * n;
                start[i]            = x4;
                start[n + i]        = __ldcg(sub.v + i);
                start[2 * n + i]    = __ldcg(sub.vprev + i);
            }
            float4 target;
            float4 const x0 = begin_substep_values<true>(sub, i, x4, target);
            if (own)
            {
                float const m = __ldg(sub.m + i);
                sub.xt[i]     = make_float4(x4.x, x4.y, x4.z, m);
                sub.xtilde[i] = target;
                T[j]          = make_float4(target.x, target.y, target.z, m / p.sweep.h2);
                if (p.sweep.kD != 0.f)
                    XT[j] = x4;
            }
            X[j] = x0;
            if constexpr (CHEB)
            {
                A[j] = x0;
                if (own)
                    B[j] = x0;
            }
            if (REC && own)
            {
                tapeX[i] = x0;
                if (word >> 31)
                    for (int k = 0; k < p.iterations; ++k)
                    {
                        tapeX[size_t(k + 1) * n + i] = x0;
                        if (CHEB)
                            tapeRaw[size_t(k) * n + i] = x0;
                    }
            }
        }
        cluster_sync<CLUSTER>();

        for (int k = 0; k < p.iterations; ++k)
        {
            float omega = 1.f;
            if constexpr (CHEB)
                omega = __ldg(p.omega + k);
            uint32_t const phase = uint32_t(ss * p.iterations + k) & 1u;
            bool const first     = ss == 0 && k == 0; // resident tiles arrive during the first iteration
            int tile             = 0; // the colour's first tile in the part
            // A warp takes the same tiles in every iteration, so that it has waited for each itself.  Once a wait
            // of the block gave up: no second arrival on a barrier whose phase did not end, and little sent to
            // blocks that stopped (they stop this one within an iteration, through what they do not send).
            if (CLUSTER)
                solving = solving && !__any_sync(0xffffffffu, *gaveUp);
            if (!solving)
            {
                for (int c = 0; c < p.nColors; ++c)
                    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
                continue;
            }
            for (int c = 0; c < p.nColors; ++c)
            {
                int2 const count       = color[c];
                uint32_t const expects = uint32_t(count.y) * (CHEB ? 32u : 16u);
                if (CLUSTER && threadIdx.x == 0 && expects)
                    barrier_expect(halo + c, expects);
                int const groups = (count.x * L + 31) / 32; // one warp each
                for (int g = warp; g < groups; g += warps)
                {
                    int const t  = g / L;
                    int stage    = tile + t;
                    uint32_t par = 0u;
                    if (!resident)
                    {
                        stage          = stage0 + t;
                        uint32_t round = round0;
                        while (stage >= p.stages)
                        {
                            stage -= p.stages;
                            ++round;
                        }
                        par = round & 1u;
                        // The slot's last tile must be consumed first: while it is still being
                        // loaded, this parity names the phase before it, which is over.  (One phase
                        // of `empty` tells the two apart: the warp's last tile lies at most a ring
                        // back, stages >= warps / L, so the tile two rings back is consumed.)
                        if (round > 0u)
                            solving = solving && barrier_wait(empty + stage, (round - 1u) & 1u, gaveUp, flags, ns);
                    }
                    if (!resident || first)
                    {
                        solving = __all_sync(0xffffffffu, solving && barrier_wait(full + stage, par, gaveUp, flags, ns));
                        if (!solving)
                            break;
                    }
                    unsigned char const* const base = ring + size_t(stage) * size_t(p.stageBytes);
                    int4 const* const entry         = reinterpret_cast<int4 const*>(base) + 2 * ((g % L) * (32 / L) + wlane / L);
                    int4 const e0                   = entry[0];
                    int4 const e1                   = entry[1];
                    bool const valid                = e0.x >= 0;
                    int const own                   = e1.x & 0xFFFF;
                    // The warp's slices follow one another from its first vertex's.
                    float4* const slice = slab + ((e0.z & 0xFFFF) - (__shfl_sync(0xffffffffu, e0.z, 0) & 0xFFFF));
                    VertexBlock<float> b;
                    zero(b);
                    float xi[3] = {0.f, 0.f, 0.f};
                    if (valid)
                    {
                        uint2 const* const nbr = reinterpret_cast<uint2 const*>(base) + (e0.z & 0xFFFF);
                        int const nNbr         = int(uint32_t(e0.z) >> 16);
                        load3(A[own], xi);
                        for (int j = lane; j < nNbr; j += kNbrs * L)
                        {
                            uint2 a[kNbrs];
                            float4 xa[kNbrs];
#pragma unroll
                            for (int u = 0; u < kNbrs; ++u)
                                a[u] = nbr[min(j + u * L, nNbr - 1)];
#pragma unroll
                            for (int u = 0; u < kNbrs; ++u)
                                xa[u] = (CHEB && !(a[u].x >> 31) ? A : X)[a[u].x & 0x7FFFu];
#pragma unroll
                            for (int u = 0; u < kNbrs; ++u)
                                if (j + u * L < nNbr)
                                    stage_neighbour(b, slice + j + u * L, xa[u], xi, __uint_as_float(a[u].y));
                        }
                    }
                    __syncwarp();
                    if (valid)
                    {
                        float4 const* const mat     = reinterpret_cast<float4 const*>(base) + (e0.w & 0xFFFF);
                        uint32_t const* const slots = reinterpret_cast<uint32_t const*>(base) + (e1.y & 0xFFFF);
                        int const nPair             = int(uint32_t(e0.w) >> 16);
                        for (int j = lane; j < nPair; j += L)
                            staged_pair(b, slice, slots[j], mat[j]);
                    }
                    reduce_lanes<L>(b);
                    if (valid && lane == 0)
                    {
                        float4 const t4   = T[own];
                        float const xl[3] = {t4.x, t4.y, t4.z};
                        float xt[3]       = {0.f, 0.f, 0.f};
                        if (p.sweep.kD != 0.f)
                            load3(XT[own], xt);
                        b.s = __int_as_float(e1.z);
                        float H[6], gr[3];
                        elastic_system(b, xt, xi, p.sweep.h, p.sweep.kD, H, gr);
                        bool const moved = inertia_solve(H, gr, xl, t4.w, p.sweep.detHZero, xi);
                        if constexpr (REC)
                            store_inverse(H, moved, tapeH + (size_t(k) * size_t(p.nFree) + size_t(e0.y)) * 2);
                        float4 const raw = make_float4(xi[0], xi[1], xi[2], 0.f);
                        float4 acc       = raw;
                        X[own]           = raw;
                        if constexpr (CHEB)
                        {
                            if (k > 1)
                            {
                                float4 const km2 = B[own];
                                acc.x            = omega * (xi[0] - km2.x) + km2.x;
                                acc.y            = omega * (xi[1] - km2.y) + km2.y;
                                acc.z            = omega * (xi[2] - km2.z) + km2.z;
                            }
                            B[own] = A[own];
                            A[own] = acc;
                        }
                        if constexpr (REC)
                        {
                            tapeX[size_t(k + 1) * n + size_t(e0.x)] = acc;
                            if (CHEB)
                                tapeRaw[size_t(k) * n + size_t(e0.x)] = raw;
                        }
                        if constexpr (CLUSTER)
                        {
                            uint32_t const* const copies = reinterpret_cast<uint32_t const*>(base) + (uint32_t(e1.y) >> 16);
                            int const nCopies            = int(uint32_t(e1.x) >> 16);
#pragma unroll 1
                            for (int q = 0; q < nCopies; ++q)
                            {
                                uint32_t const to  = copies[q];
                                uint32_t const bar = remote_address(shared_address(halo + c), to >> 16);
                                store_async(remote_address(shared_address(X + (to & 0xFFFFu)), to >> 16), bar, raw);
                                if (CHEB)
                                    store_async(remote_address(shared_address(A + (to & 0xFFFFu)), to >> 16), bar, acc);
                            }
                        }
                    }
                    __syncwarp();
                    if (!resident && wlane == 0)
                        barrier_arrive(empty + stage, g + 1 == groups ? uint32_t(L - g % L) : 1u);
                }
                int const colorTiles = (count.x + kClusterTileVertices - 1) / kClusterTileVertices;
                tile += colorTiles;
                stage0 += colorTiles;
                while (stage0 >= p.stages)
                {
                    stage0 -= p.stages;
                    ++round0;
                }
                // One warp, the one with the least to solve, waits for the block: its acquire empties the SM's L1,
                // and the block's barrier passes on what it makes visible.
                if (CLUSTER && expects && warp == warps - 1)
                    barrier_wait<true>(halo + c, phase, gaveUp, flags, ns);
                asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
            }
        }

        for (int j = int(threadIdx.x); j < nOwned; j += threads)
        {
            int const i = int(__ldg(p.partVertex + v0 + j) & kIndexMask);
            end_substep_values<true>(sub, i, A[j], true);
        }
        // Before the next substep reads what other blocks wrote; and no block leaves while another may
        // still store to it (one whose wait gave up).
        if (CLUSTER || ss + 1 < p.substeps)
            cluster_sync<CLUSTER>();
    }
    // Positions sent to a block that stopped waiting for them may still be on their way (a microsecond or
    // so; there is no barrier left to tell): it stays until long after.
    if (CLUSTER && *gaveUp)
        for (int n = 0; n < 100; ++n)
            __nanosleep(1000);
}

template <bool CHEB, bool REC, bool CLUSTER>
void const* kernel_l(int lanes)
{
    switch (lanes)
    {
        case 1: return reinterpret_cast<void const*>(cluster_step_kernel<1, CHEB, REC, CLUSTER>);
        case 2: return reinterpret_cast<void const*>(cluster_step_kernel<2, CHEB, REC, CLUSTER>);
        case 4: return reinterpret_cast<void const*>(cluster_step_kernel<4, CHEB, REC, CLUSTER>);
        case 8: return reinterpret_cast<void const*>(cluster_step_kernel<8, CHEB, REC, CLUSTER>);
        case 16: return reinterpret_cast<void const*>(cluster_step_kernel<16, CHEB, REC, CLUSTER>);
        case 32: return reinterpret_cast<void const*>(cluster_step_kernel<32, CHEB, REC, CLUSTER>);
        default: return nullptr;
    }
}

void const* kernel_of(int lanes, bool cheb, bool rec, bool cluster)
{
    if (cluster)
        return cheb ? (rec ? kernel_l<true, true, true>(lanes) : kernel_l<true, false, true>(lanes))
                    : (rec ? kernel_l<false, true, true>(lanes) : kernel_l<false, false, true>(lanes));
    return cheb ? (rec ? kernel_l<true, true, false>(lanes) : kernel_l<true, false, false>(lanes))
                : (rec ? kernel_l<false, true, false>(lanes) : kernel_l<false, false, false>(lanes));
}

void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int warps, int blocks, int nMeshes, size_t smem, cudaStream_t s)
{
    cfg.gridDim          = dim3(unsigned(blocks) * unsigned(nMeshes));
    cfg.blockDim         = dim3(unsigned(32 * (warps + 1)));
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = s;
    cfg.attrs            = attr;
    cfg.numAttrs         = 0;
    if (blocks > 1)
    {
        attr[0].id               = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = unsigned(blocks);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.numAttrs             = 1;
    }
}

} // namespace

size_t cluster_step_smem(ClusterStepParams const& p, int warps, bool chebyshev)
{
    size_t const positions = (chebyshev ? 2 * size_t(p.localCapacity) + size_t(p.ownedCapacity) : size_t(p.localCapacity)) +
                             (p.sweep.kD != 0.f ? size_t(p.ownedCapacity) : 0);
    return size_t(p.stages) * size_t(p.stageBytes) + 2 * (size_t(p.stages) + size_t(p.nColors)) * sizeof(uint64_t) +
           (positions + size_t(p.ownedCapacity) + size_t(p.slabPerWarp) * size_t(warps)) * sizeof(float4);
}

cudaError_t launch_cluster_step(ClusterStepParams const& p, int lanes, int warps, int blocks, int nMeshes, bool chebyshev, bool record, cudaStream_t s)
{
    void const* k     = kernel_of(lanes, chebyshev, record, blocks > 1);
    size_t const smem = cluster_step_smem(p, warps, chebyshev);
    if (!k || nMeshes < 1 || blocks < 1 || blocks > kClusterMaxBlocks || warps < 1 || warps > kClusterMaxWarps || p.stages < 1 ||
        p.stages > kClusterMaxStages || p.stages * lanes < warps || p.stageBytes % 128 != 0 || smem > kClusterMaxBytes)
        return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    configure(cfg, attr, warps, blocks, nMeshes, smem, s);
    ClusterStepParams q = p;
    void* args[]        = {&q};
    return cudaLaunchKernelExC(&cfg, k, args);
}

int cluster_step_resident(int lanes, int warps, int blocks, size_t smem, bool chebyshev, bool record)
{
    void const* k = kernel_of(lanes, chebyshev, record, blocks > 1);
    int n         = 0;
    bool ok       = k && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kClusterMaxBytes)) == cudaSuccess;
    if (ok && blocks > 8)
        ok = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (ok)
    {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        configure(cfg, attr, warps, blocks, 1, smem, nullptr);
        ok = blocks > 1 ? cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess
                        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 32 * (warps + 1), smem) == cudaSuccess;
    }
    if (!ok)
        cudaGetLastError();
    return ok ? n : 0;
}

} // namespace pbgb
