// Adjoint of the VBD step (no reference counterpart: the reference has no differentiation).
//
// A recorded substep keeps, for iterations k = 0..K, the iterate X_k after iteration k (X_0: the
// initial guess) and, per iteration and solved vertex, the inverse of the vertex's 3x3 Newton
// matrix.  Reversing the substep runs the colour sweeps backwards (iterations K..1, colours last
// to first).  Reversing colour c of iteration k is the same block sweep on the transposed system:
// every vertex o of the colour forms w = H^-1 u from its adjoint u, then each incident tet adds
// -d(phi)/dx to the adjoints of its three other corners (atomics: those belong to other colours)
// and to o's own, with phi = w . (g - H delta) (adjoint_tet in vbd_math.cuh).  The state a vertex
// saw before its update is rebuilt from the tape by the colour rank bits of the tet record: a
// corner of lower rank from X_k, one of higher rank (and o itself) from X_{k-1}.
//
// Rayleigh damping (D = kD / h) makes the Newton matrix (1 + D) H_e + K I and adds D H_e (x_o - xt_o)
// to the gradient, so the tet terms use delta' = (1 + D) delta - D (x_o - xt_o), the own vertex
// loses D H_e w = D (u - K w) / (1 + D) more, and xt_o gains it.  Chebyshev (y_k = omega (raw_k -
// y_{k-2}) + y_{k-2}) is reversed by splitting each iterate's adjoint between its raw sweep result
// and the iterate two back (launch_adjoint_cheb_mix), the reversed sweep reading raw_k for lower
// colours and y_{k-1} for its own and higher colours.  The initial guess enters through
// launch_adjoint_end, including the derivative of the adaptive guesses' acceleration factor on the
// branch the forward took.
//
// Not supported: contact, Anderson, Nesterov, Broyden and trust-region acceleration.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vbd_kernels.cuh"

namespace pbgb {

struct AdjointSweepParams
{
    float4 const* __restrict__ xk;   // X_k
    float4 const* __restrict__ xkm1; // X_{k-1}
    float4 const* __restrict__ X;    // rest positions
    TetRecord const* __restrict__ tets;
    int32_t const* __restrict__ solve;
    int32_t const* __restrict__ incPtr;
    uint32_t const* __restrict__ inc;
    float4 const* __restrict__ tape; // inverse Newton matrices of iteration k (2 float4 per entry)
    float const* __restrict__ m;     // lumped masses
    float4* __restrict__ ubar;       // adjoint of the positions (in: after the colour, out: before)
    float4* __restrict__ xtbar;      // adjoint of the inertial target, accumulated
    // Per tet, accumulated in FP64: each is a sum over every iteration of terms that largely
    // cancel (about 4 x iterations x steps of them), which FP32 accumulation does not resolve.
    double* __restrict__ dlogmu;
    double* __restrict__ dloglambda;
    // Damping: D = kD / h (0: none), xs = the substep's start positions, xsbar = their adjoint
    // through the damping term (accumulated).
    float4 const* __restrict__ xs;
    float4* __restrict__ xsbar;
    float D;
    int32_t begin;
    int32_t end;
    float h2;
};

// pdl: programmatic dependent launch (the kernel waits before reading the adjoints).
cudaError_t launch_adjoint_sweep(AdjointSweepParams const& p, int lanes, int block, bool pdl, cudaStream_t s);

// The reversed substep of a small mesh, in three kernels instead of a launch per colour and iteration:
//
//  * blocks: what an update of o adds to the adjoint of a neighbour j is linear in w_o, with a 3x3 block
//    that only the tape decides.  All blocks of several iterations are formed at once, one lane per edge
//    (o, j) over the tets around it, and their sum per o, the own adjoint's;
//  * chain: the iterations and colours in turn, in one block.  A vertex gathers the blocks
//    of its solved neighbours times their w -- of higher colours, which this iteration has formed, and of
//    lower colours, from the iteration reversed before -- then forms its own w and keeps it.  No adjoint
//    is added to by another vertex: no atomics, and the same bits in every run;
//  * material: the sensitivities of every tet, linear in w too, from the kept w of all iterations.
//
// In the scatter (launch_adjoint_sweep) each colour waits for the previous one's launch, the tets'
// arithmetic and its atomics: 4.3 us a colour and iteration, the chain 1.2 us (81 vertices).
struct AdjointChain
{
    // Edges (o, j) by solve entry o: entries edgePtr[s] .. edgePtr[s + 1], each with its place in j's
    // gather list and its tets, incidence codes tet << 4 | corner of o << 2 | index of j among the others.
    int32_t const* edgePtr;
    int32_t const* edgePlace;
    int32_t const* tetPtr; // per edge
    uint32_t const* tetCode;
    // Gather lists by vertex j: solve entries of the neighbours, higher colours in gatherPtr[j] ..
    // gatherMid[j], lower ones (all of them for a vertex that is never solved) up to gatherPtr[j + 1].
    // gatherAt: their places in the chain's shared memory.
    int32_t const* gatherPtr;
    int32_t const* gatherMid;
    int32_t const* gather;
    int32_t const* gatherAt;
    int32_t const* solve;
    int32_t const* fixed; // the vertices that are never solved
    int32_t const* entry; // solve entry of a vertex, -1: never solved
    int32_t const* colorPtr;
    float4 const* X;
    TetRecord const* tets;
    float const* m;
    // Tape: iterate k at x + k nV, raw sweep result at raw + k nV, inverse matrices at tape + 2 k nFree.
    float4 const* x;
    float4 const* raw;
    float4 const* tape;
    float4 const* xs;
    // Per iteration from kLo: block rows (2 float4 and a float per gather entry) and own sums (3 float4
    // per solve entry); w of every iteration.
    float4* block0;
    float4* block1;
    float* block2;
    float4* own;
    float4* w;
    float4* ubar;
    float4* xtbar;
    float4* xsbar;
    float4* yp;  // Chebyshev carries, nullptr without
    float4* ypp;
    float const* omega; // Chebyshev weights per iteration
    double* dlogmu;
    double* dloglambda;
    int32_t nV, nT, nFree, nFixed, nEdges, nColors, iterations;
    int32_t kLo, kHi;
    float D, h2;
};

int constexpr kAdjointChainThreads = 512, kAdjointChainLanes = 8, kAdjointChainAhead = 2, kAdjointChainColors = 64;
int constexpr kAdjointChainGroups = kAdjointChainThreads / kAdjointChainLanes;
size_t constexpr kAdjointChainMaxBytes = 200 * 1024;

cudaError_t launch_adjoint_blocks(AdjointChain const& p, cudaStream_t s);
// Iterations kHi - 1 .. kLo in one block of `groups` groups of lanes, a multiple of 4 and at least the
// largest colour, with smem bytes of shared memory (adjoint_chain_smem).
cudaError_t launch_adjoint_chain(AdjointChain const& p, int groups, size_t smem, cudaStream_t s);
size_t adjoint_chain_smem(int nColors, int groups, bool chebyshev);
// Whether a block has that much; also prepares the kernel for it.
bool adjoint_chain_fits(size_t smem);
cudaError_t launch_adjoint_material(AdjointChain const& p, cudaStream_t s);

// Start of a reversed substep: ubar = xbar + vbar / h (v = (x - xt)/h), xtbar = xsbar = 0, and the
// Chebyshev carries yp = ypp = 0 (nullable).
cudaError_t launch_adjoint_begin(int32_t n, float const* xbar, float const* vbar, float4* ubar, float4* xtbar, float4* xsbar,
                                 float4* yp, float4* ypp, float h, cudaStream_t s);

// Before reversing Chebyshev iteration k: y = yp + ubar (the complete adjoint of y_k), ubar = c1 y
// (raw_k's), yp = ypp (y_{k-1}'s so far), ypp = c2 y (y_{k-2}'s); c1 = omega_k, c2 = 1 - omega_k for
// k > 1, else 1 and 0.
cudaError_t launch_adjoint_cheb_mix(int32_t n, float4* ubar, float4* yp, float4* ypp, float c1, float c2, cudaStream_t s);

// End of a reversed substep: the adjoints of the substep's start positions, velocities and
// previous velocities, in place of xbar, vbar and pbar (n x 3 each).  With xtilde = xt + h v + h^2 a,
// the initial guess x0 = xt + s1 h v + h^2 a_t(v, vtm1) a (vtm1: the previous velocity with GPU
// semantics, v otherwise) and the next previous velocity = v (GPU semantics):
//   xbar <- -vbar/h + ubar + xtbar + xsbar
//   vbar <- s1 h ubar + h xtbar + h^2 (a . ubar) da_t/dv + [GPU] pbar
//   pbar <- h^2 (a . ubar) da_t/dvtm1
// v0, p0, a: the substep's start velocities, previous velocities and external accelerations.
cudaError_t launch_adjoint_end(int32_t n, float* xbar, float* vbar, float* pbar, float4 const* ubar, float4 const* xtbar,
                               float4 const* xsbar, float4 const* v0, float4 const* p0, float4 const* a, float h,
                               int32_t strategy, int32_t gpuSemantics, cudaStream_t s);

} // namespace pbgb
