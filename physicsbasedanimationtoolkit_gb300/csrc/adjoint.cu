// Adjoint sweep kernels (see adjoint.cuh).
#include "adjoint.cuh"

#include <cfloat>

namespace pbgb {

namespace {

__device__ __forceinline__ uint32_t corner_of(uint4 const& t, int a)
{
    return a == 0 ? t.x : (a == 1 ? t.y : (a == 2 ? t.z : t.w));
}

// One incidence of the reversed vertex: its tet, the three other corners' positions as the vertex
// saw them (lower colour rank: X_k, higher: X_{k-1}) relative to o's, and the rest edges.
struct AdjointIncidence
{
    int e;
    float4 mat;
    int j[3];
    float d[3][3];
    float E[3][3];
};

__device__ __forceinline__ void load_incidence(AdjointSweepParams const& p, uint32_t q, float4 const& pre, float4 const& Xo, AdjointIncidence& a)
{
    a.e                = int(q >> 2);
    int const il       = int(q & 3u);
    TetRecord const r  = p.tets[a.e];
    a.mat              = r.mat;
    uint32_t const rnk = corner_of(r.v, il) >> 30;
#pragma unroll
    for (int m = 0; m < 3; ++m)
    {
        uint32_t const ta = corner_of(r.v, (il + 1 + m) & 3);
        a.j[m]            = int(ta & kIndexMask);
        float4 const xa   = (ta >> 30) < rnk ? p.xk[a.j[m]] : p.xkm1[a.j[m]];
        float4 const Xa   = p.X[a.j[m]];
        a.d[m][0] = xa.x - pre.x, a.d[m][1] = xa.y - pre.y, a.d[m][2] = xa.z - pre.z;
        a.E[m][0] = Xa.x - Xo.x, a.E[m][1] = Xa.y - Xo.y, a.E[m][2] = Xa.z - Xo.z;
    }
}

// L lanes per vertex o of the colour, as in the forward sweep: lane l takes incidences l, l+L, ...
// Everything but o's own adjoint comes from the tape and the mesh tables, which no launch of the
// reversed step writes: the vertex's tape entries, its lane's first incidence and that
// incidence's w-independent terms (adjoint_tet_prepare) are formed before griddepcontrol.wait, so
// that with programmatic dependent launch they overlap the previous colour's tail; the adjoint is
// read, and the neighbours' adjoints and the tets' sensitivities written, only after it.
template <int L>
__global__ void __launch_bounds__(256) adjoint_sweep_kernel(AdjointSweepParams p)
{
    int const tid    = blockIdx.x * blockDim.x + threadIdx.x;
    int const s      = p.begin + tid / L;
    int const lane   = tid & (L - 1);
    bool const valid = s < p.end;
    float own[3]     = {0.f, 0.f, 0.f};
    float w[3]       = {0.f, 0.f, 0.f};
    int i = 0, k = 0, k1 = 0;
    float4 pre = make_float4(0.f, 0.f, 0.f, 0.f), pst = pre, Xo = pre, r0 = pre, r1 = pre;
    AdjointIncidence a;
    AdjointTetPre<float> q;
    float delta[3] = {0.f, 0.f, 0.f};
    bool has = false, skipped = true;
    if (valid)
    {
        i   = p.solve[s];
        pre = p.xkm1[i];
        pst = p.xk[i];
        Xo  = p.X[i];
        r0  = p.tape[2 * s];
        r1  = p.tape[2 * s + 1];
        k   = p.incPtr[s] + lane;
        k1  = p.incPtr[s + 1];
        has = k < k1;
        // The step was skipped (singular Newton matrix, tape entry zero): x_o' = x_o, and nothing
        // else of the update depends on its inputs.
        skipped = r0.x == 0.f && r0.w == 0.f && r1.y == 0.f;
        delta[0] = pre.x - pst.x, delta[1] = pre.y - pst.y, delta[2] = pre.z - pst.z;
        if (p.D != 0.f)
        {
            float4 const xs = p.xs[i];
            delta[0]        = (1.f + p.D) * delta[0] - p.D * (pre.x - xs.x);
            delta[1]        = (1.f + p.D) * delta[1] - p.D * (pre.y - xs.y);
            delta[2]        = (1.f + p.D) * delta[2] - p.D * (pre.z - xs.z);
        }
        if (skipped)
            has = false;
        // The first incidence's w-independent terms (positions, rest state, delta: all from the
        // tape and the tables) are formed before the wait as well.
        if (has)
        {
            load_incidence(p, p.inc[k], pre, Xo, a);
            float G[3][3];
            rest_gradients(a.E, G);
            adjoint_tet_prepare(a.d, a.E, G, delta, q);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (valid)
    {
        float4 const u = p.ubar[i];
        // w = H^-1 u (symmetric: xx xy xz yy yz zz)
        w[0] = r0.x * u.x + r0.y * u.y + r0.z * u.z;
        w[1] = r0.y * u.x + r0.w * u.y + r1.x * u.z;
        w[2] = r0.z * u.x + r1.x * u.y + r1.y * u.z;
        while (has)
        {
            float c[3][3], dmu = 0.f, dla = 0.f;
            adjoint_tet_finish(q, w, delta, a.mat.x, a.mat.y, c, dmu, dla);
#pragma unroll
            for (int m = 0; m < 3; ++m)
            {
                atomicAdd(p.ubar + a.j[m], make_float4(-c[m][0], -c[m][1], -c[m][2], 0.f));
                own[0] += c[m][0];
                own[1] += c[m][1];
                own[2] += c[m][2];
            }
            // Added in L2 without a value returned: nothing here waits for the FP64 sums.
            atomicAdd(p.dlogmu + a.e, -double(dmu));
            atomicAdd(p.dloglambda + a.e, -double(dla));
            k += L;
            has = k < k1;
            if (has)
            {
                load_incidence(p, p.inc[k], pre, Xo, a);
                float G[3][3];
                rest_gradients(a.E, G);
                adjoint_tet_prepare(a.d, a.E, G, delta, q);
            }
        }
    }
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1)
#pragma unroll
        for (int r = 0; r < 3; ++r)
            own[r] += __shfl_xor_sync(0xffffffffu, own[r], off);
    if (!valid || lane != 0 || skipped)
        return;
    // d(phi)/dx_o = K w + D H_e w - sum_e (own contributions) with K = m/h^2 from the inertia term
    // and H_e w = (u - K w)/(1 + D) from the damping term.
    float const K  = p.m[i] / p.h2;
    float4 const u = p.ubar[i];
    float dHw[3]   = {0.f, 0.f, 0.f};
    if (p.D != 0.f)
    {
        float const s = p.D / (1.f + p.D);
        dHw[0]        = s * (u.x - K * w[0]);
        dHw[1]        = s * (u.y - K * w[1]);
        dHw[2]        = s * (u.z - K * w[2]);
        float4 const q = p.xsbar[i];
        p.xsbar[i]     = make_float4(q.x + dHw[0], q.y + dHw[1], q.z + dHw[2], 0.f);
    }
    p.ubar[i] = make_float4(u.x - K * w[0] - dHw[0] + own[0], u.y - K * w[1] - dHw[1] + own[1],
                            u.z - K * w[2] - dHw[2] + own[2], 0.f);
    float4 const t = p.xtbar[i];
    p.xtbar[i]     = make_float4(t.x + K * w[0], t.y + K * w[1], t.z + K * w[2], 0.f);
}

// Incidence of solve entry `o` seen from corner il of tet e, the others in the order first, first + 1,
// first + 2 of those after il: positions as o saw them relative to o's.
__device__ __forceinline__ float4 load_corners(AdjointChain const& p, int k, int e, int il, int first, float4 const& pre, float4 const& Xo, float (&d)[3][3], float (&E)[3][3])
{
    TetRecord const r  = p.tets[e];
    uint32_t const rnk = corner_of(r.v, il) >> 30;
    float4 const* xk   = p.raw + size_t(k) * size_t(p.nV);
    float4 const* xkm1 = p.x + size_t(k) * size_t(p.nV);
#pragma unroll
    for (int m = 0; m < 3; ++m)
    {
        int n             = first + m;
        n                 = n >= 3 ? n - 3 : n;
        uint32_t const ta = corner_of(r.v, (il + 1 + n) & 3);
        int const j       = int(ta & kIndexMask);
        float4 const xa   = ((ta >> 30) < rnk ? xk : xkm1)[j];
        float4 const Xa   = p.X[j];
        d[m][0] = xa.x - pre.x, d[m][1] = xa.y - pre.y, d[m][2] = xa.z - pre.z;
        E[m][0] = Xa.x - Xo.x, E[m][1] = Xa.y - Xo.y, E[m][2] = Xa.z - Xo.z;
    }
    return r.mat;
}

// The step of o in iteration k as the gradient sees it (the damped one with D).
__device__ __forceinline__ void load_delta(AdjointChain const& p, int k, int i, float4& pre, float* delta)
{
    pre              = p.x[size_t(k) * size_t(p.nV) + size_t(i)];
    float4 const pst = p.raw[size_t(k) * size_t(p.nV) + size_t(i)];
    delta[0] = pre.x - pst.x, delta[1] = pre.y - pst.y, delta[2] = pre.z - pst.z;
    if (p.D != 0.f)
    {
        float4 const xs = p.xs[i];
        delta[0]        = (1.f + p.D) * delta[0] - p.D * (pre.x - xs.x);
        delta[1]        = (1.f + p.D) * delta[1] - p.D * (pre.y - xs.y);
        delta[2]        = (1.f + p.D) * delta[2] - p.D * (pre.z - xs.z);
    }
}

int constexpr kEdgeLanes = 16;

// 16 lanes per solve entry and iteration (grid.y), an edge each at a time.
__global__ void __launch_bounds__(128) adjoint_blocks_kernel(AdjointChain p)
{
    int const s      = int(blockIdx.x * blockDim.x + threadIdx.x) / kEdgeLanes;
    int const lane   = int(threadIdx.x) & (kEdgeLanes - 1);
    int const k      = p.kLo + int(blockIdx.y);
    bool const valid = s < p.nFree;
    float sum[9];
#pragma unroll
    for (int r = 0; r < 9; ++r)
        sum[r] = 0.f;
    if (valid)
    {
        float4 const* const tape = p.tape + 2 * (size_t(k) * size_t(p.nFree) + size_t(s));
        float4 const r0 = tape[0], r1 = tape[1];
        int const i     = p.solve[s];
        float4 const Xo = p.X[i];
        float4 pre;
        float delta[3];
        load_delta(p, k, i, pre, delta);
        // A skipped step (singular Newton matrix, tape entry zero) leaves the neighbours alone.
        bool const skipped = r0.x == 0.f && r0.w == 0.f && r1.y == 0.f;
        size_t const base  = size_t(blockIdx.y) * size_t(p.nEdges);
        for (int n = p.edgePtr[s] + lane; n < p.edgePtr[s + 1]; n += kEdgeLanes)
        {
            float diag = 0.f, sy[3] = {0.f, 0.f, 0.f}, R[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}}, b[9];
            int const end = skipped ? 0 : p.tetPtr[n + 1];
            for (int t = p.tetPtr[n]; t < end; ++t)
            {
                uint32_t const q = p.tetCode[t];
                float d[3][3], E[3][3], G[3][3];
                float4 const mat = load_corners(p, k, int(q >> 4), int((q >> 2) & 3u), int(q & 3u), pre, Xo, d, E);
                rest_gradients(E, G);
                adjoint_edge(d, E, G, delta, mat.x, mat.y, diag, sy, R);
            }
            adjoint_block(diag, sy, R, b);
            size_t const at = base + size_t(p.edgePlace[n]);
            p.block0[at]    = make_float4(b[0], b[1], b[2], b[3]);
            p.block1[at]    = make_float4(b[4], b[5], b[6], b[7]);
            p.block2[at]    = b[8];
#pragma unroll
            for (int r = 0; r < 9; ++r)
                sum[r] += b[r];
        }
    }
#pragma unroll
    for (int off = kEdgeLanes / 2; off > 0; off >>= 1)
#pragma unroll
        for (int r = 0; r < 9; ++r)
            sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], off);
    if (valid && lane == 0)
    {
        float4* const own = p.own + 3 * (size_t(blockIdx.y) * size_t(p.nFree) + size_t(s));
        own[0]            = make_float4(sum[0], sum[1], sum[2], sum[3]);
        own[1]            = make_float4(sum[4], sum[5], sum[6], sum[7]);
        own[2]            = make_float4(sum[8], 0.f, 0.f, 0.f);
    }
}

// A block of a gather list, row major, its w's place (AdjointChain::gatherAt) and w.
struct ChainBlock
{
    float4 a, b;
    float e;
    int32_t at;
};

__device__ __forceinline__ void add_block(ChainBlock const& x, float4 const& w, float* acc)
{
    acc[0] += x.a.x * w.x + x.a.y * w.y + x.a.z * w.z;
    acc[1] += x.a.w * w.x + x.b.x * w.y + x.b.y * w.z;
    acc[2] += x.b.z * w.x + x.b.w * w.y + x.e * w.z;
}

// What a turn of a vertex reads that the adjoints do not decide: its first two blocks per lane and, in
// lane 0, its inverse (r0, r1), the own block (s0, s1, s2) and its mass.
struct ChainTurn
{
    int4 q;
    ChainBlock x[kAdjointChainAhead];
    float4 r0, r1, s0, s1;
    float s2, m;
};

// Bound by the colours' chain: the block's barrier, w of the neighbours from shared memory, a reduction over
// the lanes, w.  The turn's blocks and inverses are loaded one turn ahead; w, the adjoints and the carries
// stay in shared memory, and only w goes out every turn, for the sensitivities.
//
// A vertex takes what its lower neighbours of iteration k + 1 add together with what its higher ones of
// iteration k do, when its own turn comes, so that nothing happens between two iterations; the last ones
// follow at the end, and the vertices that are never solved.
__global__ void __launch_bounds__(kAdjointChainThreads) adjoint_chain_kernel(AdjointChain p)
{
    constexpr int L    = kAdjointChainLanes;
    int const perBlock = int(blockDim.x) / L; // at least the largest colour
    extern __shared__ float4 shared[];
    __shared__ int32_t color[kAdjointChainColors + 1];
    int const lane     = int(threadIdx.x) & (L - 1);
    int const local    = int(threadIdx.x) / L;
    for (int c = int(threadIdx.x); c <= p.nColors; c += int(blockDim.x))
        color[c] = p.colorPtr[c];
    __syncthreads();
    // By place (colour, group): (vertex, first, first of the lower ones, end), w of even and odd
    // iterations, adjoint, inertial target's adjoint, Chebyshev carries.
    int const places = p.nColors * perBlock;
    int4* const list = reinterpret_cast<int4*>(shared);
    float4* const W  = shared + places;
    float4* const U  = W + 2 * places;
    float4* const XT = U + places;
    float4* const Y  = XT + places;
    float4* const Z  = Y + places;
    for (int a = int(threadIdx.x); a < places; a += int(blockDim.x))
    {
        int const c = a / perBlock, s = color[c] + a % perBlock;
        list[a]     = make_int4(-1, 0, 0, 0);
        if (s < color[c + 1])
        {
            int const i = p.solve[s];
            list[a]     = make_int4(i, p.gatherPtr[i], p.gatherMid[i], p.gatherPtr[i + 1]);
            U[a]        = p.ubar[i];
            XT[a]       = p.xtbar[i];
            if (p.yp)
            {
                Y[a] = p.yp[i];
                Z[a] = p.ypp[i];
            }
        }
    }
    __syncthreads();
    auto const mix = [&](float4& y1, float4& y2, float4& u, int k) {
        float const om = p.omega[k], c1 = k > 1 ? om : 1.f, c2 = k > 1 ? 1.f - om : 0.f;
        float4 const y = make_float4(y1.x + u.x, y1.y + u.y, y1.z + u.z, 0.f);
        u              = make_float4(c1 * y.x, c1 * y.y, c1 * y.z, 0.f);
        y1             = y2;
        y2             = make_float4(c2 * y.x, c2 * y.y, c2 * y.z, 0.f);
    };
    size_t const nEdges   = size_t(p.nEdges), nFree = size_t(p.nFree);
    auto const load_block = [&](ChainBlock& x, size_t base, int t) {
        x.at = p.gatherAt[t];
        x.a  = p.block0[base + t];
        x.b  = p.block1[base + t];
        x.e  = p.block2[base + t];
    };
    auto const reduce = [](float* acc) {
#pragma unroll
        for (int off = L / 2; off > 0; off >>= 1)
#pragma unroll
            for (int r = 0; r < 3; ++r)
                acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], off);
    };
    // Lists are [higher: this iteration's w), [lower: the last one's); the lower ones of the first
    // iteration here are done.
    auto const load = [&](ChainTurn& n, int k, int c) {
        n.q          = list[c * perBlock + local];
        int const hi = k == p.kHi - 1 ? n.q.z : n.q.w;
        if (k == p.kHi - 1)
            n.q.w = n.q.z;
        size_t const base = size_t(k - p.kLo) * nEdges;
#pragma unroll
        for (int b = 0; b < kAdjointChainAhead; ++b)
        {
            int const t = n.q.y + lane + b * L;
            if (t < hi)
                load_block(n.x[b], t < n.q.z ? base : base + nEdges, t);
        }
        if (n.q.x >= 0 && lane == 0)
        {
            size_t const s     = size_t(color[c] + local);
            float4 const* tape = p.tape + 2 * (size_t(k) * nFree + s);
            float4 const* sum  = p.own + 3 * (size_t(k - p.kLo) * nFree + s);
            n.r0 = tape[0], n.r1 = tape[1];
            n.s0 = sum[0], n.s1 = sum[1], n.s2 = sum[2].x;
            n.m = p.m[n.q.x];
        }
    };
    auto const w_of = [&](ChainBlock const& x, int k) { return W[(k & 1) * places + x.at]; };
    ChainTurn even, odd;
    load(even, p.kHi - 1, p.nColors - 1);
    // One turn, and the place of the next one; the two turns' registers swap roles without a copy, which
    // would wait for the loads.
    int k = p.kHi - 1, c = p.nColors - 1;
    auto const turn = [&](ChainTurn& now, ChainTurn& next) {
        size_t const base = size_t(k - p.kLo) * nEdges;
        // The next turn's loads.
        if (c > 0)
            load(next, k, c - 1);
        else if (k > p.kLo)
            load(next, k - 1, p.nColors - 1);
        int4 const q = now.q;
        __syncthreads();
        int const place = c * perBlock + local;
        bool const mine = q.x >= 0 && lane == 0;
        bool const any  = __any_sync(0xffffffffu, q.x >= 0); // a warp without a vertex only meets the barrier
        float acc[3] = {0.f, 0.f, 0.f}, low[3] = {0.f, 0.f, 0.f};
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f), wn = u;
        if (any)
        {
#pragma unroll
            for (int b = 0; b < kAdjointChainAhead; ++b)
            {
                int const t = q.y + lane + b * L;
                if (t < q.w)
                    add_block(now.x[b], w_of(now.x[b], t < q.z ? k : k + 1), t < q.z ? acc : low);
            }
            for (int t = q.y + lane + kAdjointChainAhead * L; t < q.w; t += L)
            {
                ChainBlock y;
                load_block(y, t < q.z ? base : base + nEdges, t);
                add_block(y, w_of(y, t < q.z ? k : k + 1), t < q.z ? acc : low);
            }
            if (p.yp)
            {
                // The mix lies between the two.
                reduce(low);
                if (mine)
                {
                    u = U[place];
                    u.x -= low[0], u.y -= low[1], u.z -= low[2];
                    mix(Y[place], Z[place], u, k);
                }
            }
            else
            {
                if (mine)
                    u = U[place];
                acc[0] += low[0], acc[1] += low[1], acc[2] += low[2];
            }
            reduce(acc);
            if (mine)
            {
                u.x -= acc[0], u.y -= acc[1], u.z -= acc[2];
                // w = H^-1 u (symmetric: xx xy xz yy yz zz)
                wn.x = now.r0.x * u.x + now.r0.y * u.y + now.r0.z * u.z;
                wn.y = now.r0.y * u.x + now.r0.w * u.y + now.r1.x * u.z;
                wn.z = now.r0.z * u.x + now.r1.x * u.y + now.r1.y * u.z;
                W[(k & 1) * places + place] = wn;
            }
        }
        if (mine)
        {
            p.w[size_t(k) * nFree + size_t(color[c] + local)] = wn;
            if (!(now.r0.x == 0.f && now.r0.w == 0.f && now.r1.y == 0.f))
            {
                // As in adjoint_sweep_kernel, with the own contributions as a block.
                float const K = now.m / p.h2;
                float dHw[3]  = {0.f, 0.f, 0.f};
                if (p.D != 0.f)
                {
                    float const f  = p.D / (1.f + p.D);
                    dHw[0]         = f * (u.x - K * wn.x);
                    dHw[1]         = f * (u.y - K * wn.y);
                    dHw[2]         = f * (u.z - K * wn.z);
                    float4 const g = p.xsbar[q.x];
                    p.xsbar[q.x]   = make_float4(g.x + dHw[0], g.y + dHw[1], g.z + dHw[2], 0.f);
                }
                u.x = u.x - K * wn.x - dHw[0] + (now.s0.x * wn.x + now.s0.y * wn.y + now.s0.z * wn.z);
                u.y = u.y - K * wn.y - dHw[1] + (now.s0.w * wn.x + now.s1.x * wn.y + now.s1.y * wn.z);
                u.z = u.z - K * wn.z - dHw[2] + (now.s1.z * wn.x + now.s1.w * wn.y + now.s2 * wn.z);
                float4 const g = XT[place];
                XT[place]      = make_float4(g.x + K * wn.x, g.y + K * wn.y, g.z + K * wn.z, 0.f);
            }
            U[place] = u;
        }
        if (--c < 0)
        {
            c = p.nColors - 1;
            --k;
        }
    };
    for (;;)
    {
        turn(even, odd);
        if (k < p.kLo)
            break;
        turn(odd, even);
        if (k < p.kLo)
            break;
    }
    __syncthreads();
    // What the last iteration's lower colours add, to every vertex's own lanes, as above.
    for (int n = local; n < places; n += perBlock)
    {
        int4 const q = list[n];
        float low[3] = {0.f, 0.f, 0.f};
        for (int t = q.z + lane; t < q.w; t += L)
        {
            ChainBlock y;
            load_block(y, 0, t);
            add_block(y, w_of(y, p.kLo), low);
        }
        reduce(low);
        if (lane == 0 && q.x >= 0)
        {
            float4 const u = U[n];
            p.ubar[q.x]    = make_float4(u.x - low[0], u.y - low[1], u.z - low[2], 0.f);
            p.xtbar[q.x]   = XT[n];
            if (p.yp)
            {
                p.yp[q.x]  = Y[n];
                p.ypp[q.x] = Z[n];
            }
        }
    }
    __syncthreads(); // every w is in memory
    // Vertices that are never solved: each iteration's mix and sum in turn.
    for (int first = 0; first < p.nFixed; first += perBlock)
    {
        bool const valid = first + local < p.nFixed;
        int const j      = valid ? p.fixed[first + local] : 0;
        int const t0     = valid ? p.gatherPtr[j] : 0, t1 = valid ? p.gatherPtr[j + 1] : 0;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f), y1 = u, y2 = u;
        if (valid && lane == 0)
        {
            u = p.ubar[j];
            if (p.yp)
                y1 = p.yp[j], y2 = p.ypp[j];
        }
        float sum[3] = {0.f, 0.f, 0.f};
        for (int k = p.kHi - 1; k >= p.kLo; --k)
        {
            for (int t = t0 + lane; t < t1; t += L)
            {
                ChainBlock y;
                load_block(y, size_t(k - p.kLo) * nEdges, t);
                add_block(y, __ldcg(p.w + size_t(k) * nFree + p.gather[t]), sum);
            }
            if (p.yp || k == p.kLo)
            {
                reduce(sum);
                if (p.yp)
                    mix(y1, y2, u, k);
                u.x -= sum[0], u.y -= sum[1], u.z -= sum[2];
                sum[0] = sum[1] = sum[2] = 0.f;
            }
        }
        if (valid && lane == 0)
        {
            p.ubar[j] = u;
            if (p.yp)
                p.yp[j] = y1, p.ypp[j] = y2;
        }
    }
}

// A warp per tet: four corners times eight slices of the iterations, summed in a fixed order.
__global__ void __launch_bounds__(128) adjoint_material_kernel(AdjointChain p)
{
    int const e    = int(blockIdx.x * blockDim.x + threadIdx.x) / 32;
    int const lane = int(threadIdx.x) & 31;
    int const il   = lane & 3;
    double dmu = 0.0, dla = 0.0;
    int s = -1, i = 0;
    if (e < p.nT)
    {
        i = int(corner_of(p.tets[e].v, il) & kIndexMask);
        s = p.entry[i];
    }
    if (s >= 0)
    {
        float4 const Xo = p.X[i];
        for (int k = lane / 4; k < p.iterations; k += 8)
        {
            float4 const q = p.w[size_t(k) * size_t(p.nFree) + size_t(s)];
            if (q.x == 0.f && q.y == 0.f && q.z == 0.f)
                continue;
            float const w[3] = {q.x, q.y, q.z};
            float4 pre;
            float delta[3], d[3][3], E[3][3], G[3][3], c[3][3], a = 0.f, b = 0.f;
            load_delta(p, k, i, pre, delta);
            float4 const mat = load_corners(p, k, e, il, 0, pre, Xo, d, E);
            rest_gradients(E, G);
            AdjointTetPre<float> t;
            adjoint_tet_prepare(d, E, G, delta, t);
            adjoint_tet_finish(t, w, delta, mat.x, mat.y, c, a, b);
            dmu -= double(a);
            dla -= double(b);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
        dmu += __shfl_xor_sync(0xffffffffu, dmu, off);
        dla += __shfl_xor_sync(0xffffffffu, dla, off);
    }
    if (e < p.nT && lane == 0)
    {
        p.dlogmu[e] += dmu;
        p.dloglambda[e] += dla;
    }
}

__global__ void adjoint_begin_kernel(int32_t n, float const* __restrict__ xbar, float const* __restrict__ vbar, float4* __restrict__ ubar,
                                     float4* __restrict__ xtbar, float4* __restrict__ xsbar, float4* __restrict__ yp,
                                     float4* __restrict__ ypp, float invh)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    ubar[i] = make_float4(xbar[3 * i] + invh * vbar[3 * i], xbar[3 * i + 1] + invh * vbar[3 * i + 1],
                          xbar[3 * i + 2] + invh * vbar[3 * i + 2], 0.f);
    float4 const z = make_float4(0.f, 0.f, 0.f, 0.f);
    xtbar[i]       = z;
    xsbar[i]       = z;
    if (yp)
    {
        yp[i]  = z;
        ypp[i] = z;
    }
}

__global__ void adjoint_cheb_mix_kernel(int32_t n, float4* __restrict__ ubar, float4* __restrict__ yp, float4* __restrict__ ypp, float c1, float c2)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float4 const u = ubar[i], a = yp[i], b = ypp[i];
    float4 const y = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, 0.f);
    ubar[i]        = make_float4(c1 * y.x, c1 * y.y, c1 * y.z, 0.f);
    yp[i]          = b;
    ypp[i]         = make_float4(c2 * y.x, c2 * y.y, c2 * y.z, 0.f);
}

__global__ void adjoint_end_kernel(int32_t n, float* __restrict__ xbar, float* __restrict__ vbar, float* __restrict__ pbar,
                                   float4 const* __restrict__ ubar, float4 const* __restrict__ xtbar,
                                   float4 const* __restrict__ xsbar, float4 const* __restrict__ v0,
                                   float4 const* __restrict__ p0, float4 const* __restrict__ a0, float h,
                                   int32_t strategy, int32_t gpuSemantics)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float const invh  = 1.f / h;
    float const s1    = strategy == 0 ? 0.f : 1.f;
    float4 const u    = ubar[i];
    float4 const t    = xtbar[i];
    float4 const q    = xsbar[i];
    float4 const v4   = v0[i];
    float4 const a4   = a0[i];
    float4 const m4   = gpuSemantics ? p0[i] : v4;
    float const uu[3] = {u.x, u.y, u.z};
    float const tt[3] = {t.x, t.y, t.z};
    float const qq[3] = {q.x, q.y, q.z};
    float const vt[3] = {v4.x, v4.y, v4.z};
    float const vm[3] = {m4.x, m4.y, m4.z};
    float const a[3]  = {a4.x, a4.y, a4.z};
    float dAv[3], dAvm[3];
    initial_position_factor_derivatives(vm, vt, a, h, strategy, FLT_MIN, dAv, dAvm);
    float const au = a[0] * uu[0] + a[1] * uu[1] + a[2] * uu[2];
    for (int r = 0; r < 3; ++r)
    {
        float const vb  = vbar[3 * i + r];
        float const pb  = pbar[3 * i + r];
        xbar[3 * i + r] = -invh * vb + uu[r] + tt[r] + qq[r];
        vbar[3 * i + r] = s1 * h * uu[r] + h * tt[r] + h * h * au * dAv[r] + (gpuSemantics ? pb : 0.f);
        pbar[3 * i + r] = h * h * au * dAvm[r];
    }
}

inline int blocks_of(int64_t n, int b)
{
    return int((n + b - 1) / b);
}

template <int L>
cudaError_t launch_l(AdjointSweepParams const& p, int block, bool pdl, cudaStream_t s)
{
    int64_t const n        = int64_t(p.end - p.begin) * L;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim            = dim3(unsigned(blocks_of(n, block)));
    cfg.blockDim           = dim3(unsigned(block));
    cfg.stream             = s;
    cudaLaunchAttribute attr[1];
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs                                          = attr;
    cfg.numAttrs                                       = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, adjoint_sweep_kernel<L>, p);
}

} // namespace

cudaError_t launch_adjoint_sweep(AdjointSweepParams const& p, int lanes, int block, bool pdl, cudaStream_t s)
{
    if (p.end <= p.begin)
        return cudaSuccess;
    if (block <= 0 || block > 256 || block % 32 != 0)
        return cudaErrorInvalidValue;
    switch (lanes)
    {
        case 1: return launch_l<1>(p, block, pdl, s);
        case 2: return launch_l<2>(p, block, pdl, s);
        case 4: return launch_l<4>(p, block, pdl, s);
        case 8: return launch_l<8>(p, block, pdl, s);
        case 16: return launch_l<16>(p, block, pdl, s);
        case 32: return launch_l<32>(p, block, pdl, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_adjoint_blocks(AdjointChain const& p, cudaStream_t s)
{
    if (p.nFree <= 0 || p.kHi <= p.kLo)
        return cudaSuccess;
    adjoint_blocks_kernel<<<dim3(unsigned(blocks_of(int64_t(p.nFree) * kEdgeLanes, 128)), unsigned(p.kHi - p.kLo)), 128, 0, s>>>(p);
    return cudaGetLastError();
}

size_t adjoint_chain_smem(int nColors, int groups, bool chebyshev)
{
    return size_t(nColors) * size_t(groups) * sizeof(float4) * (chebyshev ? 7 : 5);
}

bool adjoint_chain_fits(size_t smem)
{
    if (smem > kAdjointChainMaxBytes)
        return false;
    if (cudaFuncSetAttribute(adjoint_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kAdjointChainMaxBytes)) == cudaSuccess)
        return true;
    cudaGetLastError();
    return false;
}

cudaError_t launch_adjoint_chain(AdjointChain const& p, int groups, size_t smem, cudaStream_t s)
{
    if (p.kHi <= p.kLo || p.nV <= 0)
        return cudaSuccess;
    if (groups < 4 || groups > kAdjointChainGroups || groups % 4 || p.nColors < 1 || p.nColors > kAdjointChainColors || smem > kAdjointChainMaxBytes)
        return cudaErrorInvalidValue;
    adjoint_chain_kernel<<<1, groups * kAdjointChainLanes, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_material(AdjointChain const& p, cudaStream_t s)
{
    if (p.nT <= 0 || p.iterations <= 0)
        return cudaSuccess;
    adjoint_material_kernel<<<blocks_of(32 * int64_t(p.nT), 128), 128, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_begin(int32_t n, float const* xbar, float const* vbar, float4* ubar, float4* xtbar, float4* xsbar,
                                 float4* yp, float4* ypp, float h, cudaStream_t s)
{
    if (n <= 0)
        return cudaSuccess;
    if ((yp == nullptr) != (ypp == nullptr))
        return cudaErrorInvalidValue;
    adjoint_begin_kernel<<<blocks_of(n, 256), 256, 0, s>>>(n, xbar, vbar, ubar, xtbar, xsbar, yp, ypp, 1.f / h);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_cheb_mix(int32_t n, float4* ubar, float4* yp, float4* ypp, float c1, float c2, cudaStream_t s)
{
    if (n <= 0)
        return cudaSuccess;
    adjoint_cheb_mix_kernel<<<blocks_of(n, 256), 256, 0, s>>>(n, ubar, yp, ypp, c1, c2);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_end(int32_t n, float* xbar, float* vbar, float* pbar, float4 const* ubar, float4 const* xtbar,
                               float4 const* xsbar, float4 const* v0, float4 const* p0, float4 const* a, float h,
                               int32_t strategy, int32_t gpuSemantics, cudaStream_t s)
{
    if (n <= 0)
        return cudaSuccess;
    adjoint_end_kernel<<<blocks_of(n, 256), 256, 0, s>>>(n, xbar, vbar, pbar, ubar, xtbar, xsbar, v0, p0, a, h, strategy,
                                                         gpuSemantics);
    return cudaGetLastError();
}

} // namespace pbgb
