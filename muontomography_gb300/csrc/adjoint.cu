// Adjoint of the MLSD negative log-likelihood plus the MAP prior with respect
// to log(lambda).  Not in the reference; it differentiates the model whose EM
// and MAP updates the reference implements:
//   NLL(l)   = sum_i log det Sigma_i + 1/2 sum_planes v^T Sigma_i^-1 v
//              (the per-muon cost of src/MutoMLSD.cpp:465-468)
//   dNLL/dl_j = sum_i pr^2 (tr(Sigma_i^-1 W_ij) - 1/2 xyS_ij) = -sum_i g_ij,
//              summed per voxel by the voxel pass in gradient mode (em_voxel.cu).
//   prior    = 2 beta sum_j sum_{m in N(j)} w_jm psi(l_j - l_m) [+ 2 beta sum_j psi(l_j)],
//              psi(t) = (t^2 + delta^2)^(p/2), l = 1e7 lambda, stencil and edge
//              clamping of src/MutoMAP.cpp:283-350: the penalty whose separable
//              surrogate is minimised by the MAP step (src/MutoMAP.cpp:207-281).
// A stencil term moves both of its voxels.  Its other voxel has the same term
// from its own side (the offset negated where it was not clamped, kept where it
// was; as many axes, so the same weight), so a voxel's derivative is twice the sum
// over its own terms, also at clamped edges.
#include "common.cuh"

namespace muto {
namespace {

inline unsigned blocks_for(uint64_t n, int threads) {
    const uint64_t b = (n + threads - 1) / threads;
    return static_cast<unsigned>(b > 0 ? b : 1);
}

// lambda in FP64 and, in the mixed form, in FP32 from one exponential
template <typename Real>
__global__ void k_exp_lambda(const double* __restrict__ loglam, const uint32_t* __restrict__ mult, uint32_t V,
                             double* __restrict__ lam64, Real* __restrict__ lam) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= V) return;
    const double v = mult[j] > 0 ? exp(loglam[j]) : 0.0;
    lam64[j] = v;
    if (lam) lam[j] = static_cast<Real>(v);
}

// The prior's value, and grad_j += l_j dF/dl_j of every voxel with pairs (chain
// rule through l = 1e7 exp(x)).  FP64 work bounds it: 26 neighbours a voxel at two
// FP64 lanes a clock and SM.  So a term costs as few FP64 operations as it can:
// sums per kind of neighbour (faces, edges, corners), weighted and scaled once at
// the end, and for p = 2 a difference, its sum and its square's sum alone.  A
// voxel's terms are gathered, not scattered with an FP64 reduction each, and a block
// adds its value once.  96 x 96 x 48 voxels, 26 neighbours,
// p = 2: 86 us (its FP64 operations alone take 75); 295 us with the terms scattered.
// Blocks are as small as it takes for every SM to have one (down to a warp): a few
// large ones leave the FP64 pipes of most SMs idle (16^3 voxels, p = 1.5: the objective
// takes 184 us, 261 with 256 threads).
constexpr int kPriorThreads = 256;  // at most
template <int POWER>
__global__ void __launch_bounds__(kPriorThreads) k_prior(const double* __restrict__ lam64,
                                                         const uint32_t* __restrict__ mult, DevGrid g, MapParams mp,
                                                         double* __restrict__ grad, double* __restrict__ value) {
    const uint32_t nx = g.n[0], ny = g.n[1], nz = g.n[2], nxy = nx * ny;
    const uint32_t V = nxy * nz;
    const double unit = 1.0e7, d2 = mp.delta * mp.delta, e = (mp.p - 2.0) / 2.0;
    const double w2 = 0.70710678118654752440, w3 = 0.57735026918962576451;  // 1/sqrt(2), 1/sqrt(3)
    const double scale = POWER == kMapTwo ? unit : 1.0;                     // of the differences summed below
    double v = 0.0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < V;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t j = static_cast<uint32_t>(i);
        const uint32_t x = j % nxy % nx, y = j % nxy / nx, z = j / nxy;
        const uint32_t xs[3] = {0 < x ? x - 1 : 0, x, x < nx - 1 ? x + 1 : nx - 1};
        const uint32_t ys[3] = {0 < y ? y - 1 : 0, y, y < ny - 1 ? y + 1 : ny - 1};
        const uint32_t zs[3] = {0 < z ? z - 1 : 0, z, z < nz - 1 ? z + 1 : nz - 1};
        const double lj = lam64[j];
        double Q[3], S[3];  // per kind: sum psi (for p = 2 without its delta^2), sum t q
#pragma unroll
        for (int k = 0; k < 3; ++k) Q[k] = S[k] = 0.0;
#pragma unroll
        for (int c = 0; c < 27; ++c) {
            const int ox = c % 3 - 1, oy = (c / 3) % 3 - 1, oz = c / 9 - 1;
            const int kind = (ox != 0) + (oy != 0) + (oz != 0) - 1;
            if (kind < 0 || (kind > 0 && !mp.all_neighbours)) continue;
            const double d = lj - lam64[xs[ox + 1] + ys[oy + 1] * nx + zs[oz + 1] * nxy];
            if (POWER == kMapTwo) {
                S[kind] += d;
                Q[kind] = fma(d, d, Q[kind]);
            } else {
                const double t = d * unit, u = fma(t, t, d2), q = map_q<POWER>(u, e);
                S[kind] = fma(t, q, S[kind]);
                Q[kind] = fma(u, q, Q[kind]);
            }
        }
        double own = fma(w3, S[2], fma(w2, S[1], S[0])) * (2.0 * scale);
        double psi = fma(w3, Q[2], fma(w2, Q[1], Q[0])) * (scale * scale);
        if (POWER == kMapTwo) psi = fma(mp.all_neighbours ? 6.0 + 12.0 * w2 + 8.0 * w3 : 6.0, d2, psi);
        if (mp.add_object_prior) {
            const double t = lj * unit, u = fma(t, t, d2), q = map_q<POWER>(u, e);
            own = fma(t, q, own);
            psi = fma(u, q, psi);
        }
        v = fma(2.0 * mp.beta, psi, v);
        if (grad && mult[j] > 0) grad[j] = fma(lj * unit * (2.0 * mp.beta * mp.p), own, grad[j]);
    }
    __shared__ double part[kPriorThreads / 32];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = warp_sum(threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : 0.0);
        if (threadIdx.x == 0) atomicAdd(value, v);
    }
}

}  // namespace

template <typename Real>
void launch_exp_lambda(const double* loglam, const uint32_t* mult, uint32_t V, double* lam64, Real* lam, cudaStream_t s) {
    k_exp_lambda<Real><<<blocks_for(V, 256), 256, 0, s>>>(loglam, mult, V, lam64, lam); count_launches(1);
}
template void launch_exp_lambda<float>(const double*, const uint32_t*, uint32_t, double*, float*, cudaStream_t);
template void launch_exp_lambda<double>(const double*, const uint32_t*, uint32_t, double*, double*, cudaStream_t);

void launch_prior(const double* lam64, const uint32_t* mult, DevGrid g, MapParams mp, int num_sms, double* grad,
                  double* value, cudaStream_t s) {
    // blocks that loop, so that few add to the one value
    const uint64_t V = static_cast<uint64_t>(g.n[0]) * g.n[1] * g.n[2];
    int threads = kPriorThreads;
    while (threads > 32 && V < static_cast<uint64_t>(threads) * num_sms) threads /= 2;
    const unsigned need = blocks_for(V, threads);
    const unsigned nb = need < 4u * num_sms ? need : 4u * num_sms;
    if (mp.p == 2.0) k_prior<kMapTwo><<<nb, threads, 0, s>>>(lam64, mult, g, mp, grad, value);
    else if (mp.p == 1.0) k_prior<kMapOne><<<nb, threads, 0, s>>>(lam64, mult, g, mp, grad, value);
    else k_prior<kMapAny><<<nb, threads, 0, s>>>(lam64, mult, g, mp, grad, value);
    count_launches(1);
}

}  // namespace muto
