// Straight-line reconstruction (MutoSLR::reconstruct, src/MutoSLR.cpp:47-103)
// and the first pass of its iterative form (MutoSLRIter, src/MutoSLRIter.cpp:
// 15-83), one thread per ray: the incoming and outgoing lines cut at the
// grid's top and bottom planes, the Siddon walk of the straight line between
// the two points (bit-exact, as for the other methods), and per voxel the
// mean squared projected angle shared by length^2 or equally.  Sums are FP64
// atomics.  The later passes of the iterative form are order-dependent (each
// muon sees the image the muons before it left): they run over the walked
// paths level by level (k_slr_iter_steps: muons of one level share no
// voxel), or muon after muon on one warp (k_slr_iter_pass).
#include "common.cuh"
#include "geometry.cuh"

namespace muto {
namespace {

// per-ray quantities of :63-77
struct SlrRay {
    double a2;        // axz^2 + ayz^2
    double p_in[3], p_out[3];
    double l_total;   // |p_in - p_out|
};

__device__ __forceinline__ SlrRay slr_ray(const muto_ray& r, const DevGrid& g, double z_lo, double z_hi, double mag) {
    SlrRay o;
    const double axz = dmul(dsub(atan2(r.din[0], r.din[2]), atan2(r.dout[0], r.dout[2])), mag);
    const double ayz = dmul(dsub(atan2(r.din[1], r.din[2]), atan2(r.dout[1], r.dout[2])), mag);
    o.a2 = dadd(dmul(axz, axz), dmul(ayz, ayz));
    const double t_in = ddiv(dsub(z_hi, r.pin[2]), r.din[2]);
    const double t_out = ddiv(dsub(z_lo, r.pout[2]), r.dout[2]);
    double d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o.p_in[k] = dadd(r.pin[k], dmul(t_in, r.din[k]));
        o.p_out[k] = dadd(r.pout[k], dmul(t_out, r.dout[k]));
        d[k] = dsub(o.p_in[k], o.p_out[k]);
    }
    o.l_total = __dsqrt_rn(dot3(d, d));
    (void)g;
    return o;
}

// A nearly upright line (at most 1e-6 mm to the side, growing) that starts within 1e-6
// of a voxel below a grid's upper face is walked with index nx (or ny) there: the
// start's voxel is rounded up by that much (src/MutoSiddon.cpp:62-81).  Such voxels
// are outside the image: they count for the equal shares and for nothing else.
__device__ __forceinline__ bool outside(uint32_t x, uint32_t y, uint32_t z, uint32_t nx, uint32_t ny, uint32_t nz) {
    return x >= nx || y >= ny || z >= nz;
}

struct CountSink {
    uint32_t n = 0;
    __device__ void operator()(uint32_t, uint32_t, uint32_t, double) { ++n; }
};

struct SlrSink {
    double* img;
    double* weight;
    uint32_t nx, ny, nz;
    double dz, a2, l_total, share, e2;  // share: a2 / 2 / n^2 (equal shares)
    int length_weighted, has_energy;
    __device__ void operator()(uint32_t x, uint32_t y, uint32_t z, double l) {
        if (outside(x, y, z, nx, ny, nz)) return;
        const uint64_t j = static_cast<uint64_t>(x) + static_cast<uint64_t>(nx) * (y + static_cast<uint64_t>(ny) * z);
        double iv;
        if (length_weighted) {  // :80-83
            atomicAdd(weight + j, ddiv(l, dz));
            const double f = ddiv(l, l_total);
            iv = dmul(dmul(dmul(a2, 0.5), f), f);
        } else {  // :84-86
            atomicAdd(weight + j, 1.0);
            iv = share;
        }
        if (has_energy) iv = dmul(iv, e2);  // :87-89
        atomicAdd(img + j, iv);
    }
};

__global__ void k_slr(SlrArgs a, DevGrid g) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const muto_ray r = a.rays[i];
    const double z_lo = a.g.z_min;                                               // :57
    const double z_hi = dadd(a.g.z_min, dmul(a.g.dz, static_cast<double>(a.g.nz)));  // :58
    const SlrRay s = slr_ray(r, g, z_lo, z_hi, a.mag);
    double share = 0.0;
    if (!a.length_weighted) {  // the equal share needs the path's voxel count first
        CountSink c;
        siddon_walk(g, s.p_in, s.p_out, c);
        const uint64_t n = c.n;
        share = ddiv(dmul(s.a2, 0.5), static_cast<double>(n * n));
    }
    SlrSink sink{a.img, a.weight, g.n[0], g.n[1], g.n[2], a.g.dz, s.a2, s.l_total, share, dmul(r.ein, r.ein),
                 a.length_weighted, a.has_energy};
    siddon_walk(g, s.p_in, s.p_out, sink);
}

// The walked straight lines, for the in-place passes: per ray the count of its
// voxels in the image (first call) or these voxels and lengths at off[i] (second call).
struct PathSink {
    uint32_t* vox;
    double* len;
    uint32_t nx, ny, nz;
    uint32_t k = 0;
    __device__ void operator()(uint32_t x, uint32_t y, uint32_t z, double l) {
        if (outside(x, y, z, nx, ny, nz)) return;
        if (vox) {
            vox[k] = x + nx * (y + ny * z);
            len[k] = l;
        }
        ++k;
    }
};

__global__ void k_slr_paths(SlrArgs a, DevGrid g, const uint64_t* __restrict__ off, uint32_t* __restrict__ counts,
                            uint32_t* __restrict__ vox, double* __restrict__ len) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const double z_lo = a.g.z_min;
    const double z_hi = dadd(a.g.z_min, dmul(a.g.dz, static_cast<double>(a.g.nz)));
    const SlrRay s = slr_ray(a.rays[i], g, z_lo, z_hi, a.mag);
    PathSink p{off ? vox + off[i] : nullptr, off ? len + off[i] : nullptr, g.n[0], g.n[1], g.n[2]};
    siddon_walk(g, s.p_in, s.p_out, p);
    if (!off) counts[i] = p.k;
}

// The pass-independent terms of every pair, once at set-up: the weight
// increment (length / dz, or 1) and the image increment before it is scaled
// by the voxel's part of the path's sum (a^2 / 2 (length / l_total)^2, or the
// equal share a^2 / 2 / n^2), with the arithmetic of :80-89; and ein^2 per
// muon.  A thread per muon.
__global__ void k_slr_pair_terms(SlrArgs a, DevGrid g, SlrPass p) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const double z_lo = a.g.z_min;
    const double z_hi = dadd(a.g.z_min, dmul(a.g.dz, static_cast<double>(a.g.nz)));
    const muto_ray r = a.rays[i];
    const SlrRay s = slr_ray(r, g, z_lo, z_hi, a.mag);
    const uint64_t p0 = p.off[i];
    const uint32_t n = static_cast<uint32_t>(p.off[i + 1] - p0);
    double share = 0.0;
    if (!a.length_weighted) {
        CountSink c;
        siddon_walk(g, s.p_in, s.p_out, c);
        share = ddiv(dmul(s.a2, 0.5), static_cast<double>(static_cast<uint64_t>(c.n) * c.n));
    }
    for (uint32_t k = 0; k < n; ++k) {
        const double l = p.len[p0 + k];
        if (a.length_weighted) {
            p.winc[p0 + k] = ddiv(l, a.g.dz);
            const double f = ddiv(l, s.l_total);
            p.iv0[p0 + k] = dmul(dmul(dmul(s.a2, 0.5), f), f);
        } else {
            p.winc[p0 + k] = 1.0;
            p.iv0[p0 + k] = share;
        }
    }
    p.e2[i] = dmul(r.ein, r.ein);
}

// One muon of a later pass of the iterative form (src/MutoSLRIter.cpp:40-71
// with iter != 0), on one warp: the warp reads the image on the muon's path,
// sums it (lane partials, then the warp's sum), and adds to each voxel its
// increment times the voxel's part of that sum (:64-66).
// img / weight: the image and weight sums (global memory, or a copy in
// shared memory).
__device__ __forceinline__ void slr_iter_muon(const SlrArgs& a, const SlrPass& p, uint64_t i, int lane, double* img,
                                              double* weight) {
    const uint64_t p0 = p.off[i];
    const uint32_t n = static_cast<uint32_t>(p.off[i + 1] - p0);
    double part = 0.0;  // :49-52
    for (uint32_t k = lane; k < n; k += 32) part = dadd(part, img[p.vox[p0 + k]]);
    const double total = warp_sum(part);
    const double e2 = a.has_energy ? p.e2[i] : 0.0;
    for (uint32_t k = lane; k < n; k += 32) {
        const uint32_t j = p.vox[p0 + k];
        weight[j] = dadd(weight[j], p.winc[p0 + k]);
        double iv = dmul(p.iv0[p0 + k], ddiv(img[j], total));
        if (a.has_energy) iv = dmul(iv, e2);  // :87-89
        img[j] = dadd(img[j], iv);
    }
}

// A later pass muon after muon on a single warp: a muon's stores are ordered
// before the next muon's loads by __syncwarp; no other warp touches the image.
__global__ void k_slr_iter_pass(SlrArgs a, SlrPass p) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x >= 32) return;
    for (uint64_t i = 0; i < a.n; ++i) {
        slr_iter_muon(a, p, i, lane, a.img, a.weight);
        __syncwarp();
    }
}

// The pairs of every muon copied into level order: muon q of the level
// order (order[q]) gets its pairs at fo[q] .. fo[q+1], so a level's data is
// contiguous and found from the level's start alone; with ein^2 folded into the
// image increment (:87-89) and the muon's place in its step (below).  A warp per
// muon.
__global__ void k_slr_flatten(SlrPass p, const uint32_t* __restrict__ order, const uint8_t* __restrict__ place,
                              uint64_t nt, int has_energy, SlrFlat f) {
    const uint64_t q = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= nt) return;
    const uint32_t i = order[q];
    const uint64_t s0 = p.off[i], n = p.off[i + 1] - s0, d0 = f.fo[q];
    const double e2 = has_energy ? p.e2[i] : 1.0;
    for (uint64_t k = lane; k < n; k += 32) {
        f.vox[d0 + k] = p.vox[s0 + k];
        f.iv0[d0 + k] = has_energy ? dmul(p.iv0[s0 + k], e2) : p.iv0[s0 + k];
        f.winc[d0 + k] = p.winc[s0 + k];
        f.place[d0 + k] = place[q];
    }
}

// A later pass level by level.  A muon's level is one more than the highest
// level among the earlier muons that share a voxel with it, so two muons of
// one level share no voxel, and every voxel meets its muons in index order:
// each muon reads and writes the image state it would see in the sequential
// loop, whatever the order inside a level.  One block; a step is a level, or at
// most THREADS / 16 muons of a longer one.  In a step
//   sum     sixteen lanes a muon add up the image on its path (:49-52) and take
//           the sum's reciprocal;
//   pairs   a thread per pair adds its weight increment and multiplies its
//           image increment with the voxel's image (:64-66);
//   (barrier) the pair adds that product times the reciprocal to its voxel;
//   (barrier) the next step.
// Bound by the chain of a step (six FP64 operations in the sum, four with the
// conversions in the reciprocal, one after it, each about 70 cycles on this
// part's two FP64 lanes a clock per SM, two barriers) and by that pipe.  20^3
// voxels, 30 k muons, 2 449 levels: 1.29 us a step; 2.82 us with a warp a muon
// (a division a pair, a 32-lane sum a muon).  8 and 4 lanes a muon, 512 and 640
// threads took 1.29 to 1.51 us, 32 lanes 1.95.  Where the image is in global memory
// its latency bounds a step, and grids are larger and paths longer: 1 024 threads, 64
// muons a step (slr_wide).  A pass, in ms, with 384 / 768 / 1 024 threads: 32^3 with
// 50 k muons 11.7 / 9.7 / 8.9, 48^3 with 100 k 34.1 / 24.5 / 22.4, 100^3 with 100 k
// 59.6 / 38.4 / 35.0, 200^3 with 50 k 57.4 / 35.3 / 32.7 (1 024 threads with 32 lanes
// a muon: 9.2, 24.7, 41.7, 35.0); in shared memory, 20^3 with 30 k: 3.1 / 4.2 / 4.9.
// With SMEM the image and weight sums (2 V doubles) are copied into shared
// memory for the pass and back after it.  Nothing that a step loads from the
// lists depends on the image: a step's bounds are loaded five steps ahead,
// its offsets three, its pairs two.
template <bool SMEM, int THREADS>
__global__ void __launch_bounds__(THREADS) k_slr_iter_steps(SlrArgs a, SlrFlat f,
                                                            const uint32_t* __restrict__ sstart, uint32_t steps) {
    extern __shared__ double slr_smem[];
    __shared__ double s_rec[THREADS / kSlrLanes];
    constexpr int H = 32 / kSlrLanes;  // pairs of a muon's sum held per lane
    const uint32_t tid = threadIdx.x, l8 = tid % kSlrLanes, slot = tid / kSlrLanes;
    const uint32_t V = a.g.nx * a.g.ny * a.g.nz;
    double* img = a.img;
    double* weight = a.weight;
    if (SMEM) {
        img = slr_smem;
        weight = slr_smem + V;
        for (uint32_t j = tid; j < V; j += blockDim.x) {
            img[j] = a.img[j];
            weight[j] = a.weight[j];
        }
        __syncthreads();
    }
    // a step's offsets: its first pair, and counted from there this lane group's muon
    // [b, e) and the step's end q
    struct Offsets {
        uint64_t p;
        uint32_t b, e, q;
    };
    auto offsets = [&](uint32_t q0, uint32_t q1) -> Offsets {  // of the step with muons [q0, q1)
        Offsets o{0, 0, 0, 0};
        const uint32_t m = q0 + slot;
        if (q0 < q1) {
            o.p = f.fo[q0];
            o.q = static_cast<uint32_t>(f.fo[q1] - o.p);
        }
        if (m < q1) {
            o.b = static_cast<uint32_t>(f.fo[m] - o.p);
            o.e = static_cast<uint32_t>(f.fo[m + 1] - o.p);
        }
        return o;
    };
    struct Pairs {
        uint32_t v[H];  // the muon's sum
        uint32_t j;     // this thread's pair
        uint32_t place;
        double iv0, winc;
    };
    auto pairs = [&](const Offsets& o) -> Pairs {
        Pairs r{};
        const uint32_t* vox = f.vox + o.p;
#pragma unroll
        for (int h = 0; h < H; ++h)
            if (o.b + l8 + h * kSlrLanes < o.e) r.v[h] = vox[o.b + l8 + h * kSlrLanes];
        if (tid < o.q) {
            r.j = vox[tid];
            r.place = f.place[o.p + tid];
            r.iv0 = f.iv0[o.p + tid];
            r.winc = f.winc[o.p + tid];
        }
        return r;
    };
    auto first = [&](uint32_t s) -> uint32_t { return sstart[min(s, steps)]; };
    uint32_t q1 = first(1), q2 = first(2), q3 = first(3), q4 = first(4);
    Offsets o = offsets(first(0), q1), o1 = offsets(q1, q2), o2 = offsets(q2, q3);
    Pairs c = pairs(o), c1 = pairs(o1);
    for (uint32_t s = 0; s < steps; ++s) {
        if (__any_sync(kFull, o.b < o.e)) {
            double w[H];
#pragma unroll
            for (int h = 0; h < H; ++h) w[h] = o.b + l8 + h * kSlrLanes < o.e ? img[c.v[h]] : 0.0;
#pragma unroll
            for (int d = H / 2; d > 0; d >>= 1)
#pragma unroll
                for (int h = 0; h < d; ++h) w[h] = dadd(w[h], w[h + d]);
            double part = w[0];
            for (uint32_t k = o.b + l8 + H * kSlrLanes; k < o.e; k += kSlrLanes) part = dadd(part, img[f.vox[o.p + k]]);
            __syncwarp();
#pragma unroll
            for (int d = kSlrLanes / 2; d > 0; d >>= 1) part = dadd(part, __shfl_xor_sync(kFull, part, d));
            if (l8 == 0 && o.b < o.e) s_rec[slot] = reciprocal(part);
        }
        const bool mine = tid < o.q;
        double x = 0.0, inc = 0.0;
        if (mine) {
            x = img[c.j];
            inc = dmul(c.iv0, x);
            weight[c.j] = dadd(weight[c.j], c.winc);
        }
        // the lists' loads for the steps to come, while the sums' last operations run
        const Pairs c2 = pairs(o2);
        const Offsets o3 = offsets(q3, q4);
        q3 = q4;
        q4 = first(s + 5);
        __syncthreads();
        if (mine) img[c.j] = fma(inc, s_rec[c.place], x);
        for (uint32_t k = tid + THREADS; k < o.q; k += THREADS) {  // more pairs than threads
            const uint32_t j = f.vox[o.p + k];
            const double xk = img[j];
            weight[j] = dadd(weight[j], f.winc[o.p + k]);
            img[j] = fma(dmul(f.iv0[o.p + k], xk), s_rec[f.place[o.p + k]], xk);
        }
        __syncthreads();
        o = o1;
        o1 = o2;
        o2 = o3;
        c = c1;
        c1 = c2;
    }
    if (SMEM) {
        for (uint32_t j = tid; j < V; j += blockDim.x) {
            a.img[j] = img[j];
            a.weight[j] = weight[j];
        }
    }
}

}  // namespace

void launch_slr(const SlrArgs& a, cudaStream_t s) {
    if (a.n == 0) return;
    k_slr<<<static_cast<unsigned>((a.n + 127) / 128), 128, 0, s>>>(a, make_dev_grid(a.g));
    count_launches(1);
}

void launch_slr_paths(const SlrArgs& a, const uint64_t* off, uint32_t* counts, uint32_t* vox, double* len,
                      cudaStream_t s) {
    if (a.n == 0) return;
    k_slr_paths<<<static_cast<unsigned>((a.n + 127) / 128), 128, 0, s>>>(a, make_dev_grid(a.g), off, counts, vox, len);
    count_launches(1);
}

void launch_slr_pair_terms(const SlrArgs& a, const SlrPass& p, cudaStream_t s) {
    if (a.n == 0) return;
    k_slr_pair_terms<<<static_cast<unsigned>((a.n + 127) / 128), 128, 0, s>>>(a, make_dev_grid(a.g), p);
    count_launches(1);
}

void launch_slr_iter_pass(const SlrArgs& a, const SlrPass& p, cudaStream_t s) {
    if (a.n == 0) return;
    k_slr_iter_pass<<<1, 32, 0, s>>>(a, p);
    count_launches(1);
}

void launch_slr_flatten(const SlrArgs& a, const SlrPass& p, const uint32_t* order, const uint8_t* place, uint64_t nt,
                        const SlrFlat& f, cudaStream_t s) {
    if (nt == 0) return;
    k_slr_flatten<<<static_cast<unsigned>((nt * 32 + 255) / 256), 256, 0, s>>>(p, order, place, nt, a.has_energy, f);
    count_launches(1);
}

static size_t slr_shared_bytes(const muto_grid& g) {
    return 2 * sizeof(double) * static_cast<size_t>(g.nx) * g.ny * g.nz;
}

bool slr_wide(const muto_grid& g, size_t smem_optin) {
    return slr_shared_bytes(g) + kSlrStep * sizeof(double) + 1024 > smem_optin;
}

void launch_slr_iter_steps(const SlrArgs& a, const SlrFlat& f, const uint32_t* sstart, uint32_t steps, bool wide,
                           cudaStream_t s) {
    if (a.n == 0 || steps == 0) return;
    const size_t bytes = slr_shared_bytes(a.g);
    if (wide) {
        k_slr_iter_steps<false, kSlrWideStep * kSlrLanes><<<1, kSlrWideStep * kSlrLanes, 0, s>>>(a, f, sstart, steps);
    } else if (cudaFuncSetAttribute(k_slr_iter_steps<true, kSlrStep * kSlrLanes>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) == cudaSuccess) {
        k_slr_iter_steps<true, kSlrStep * kSlrLanes><<<1, kSlrStep * kSlrLanes, bytes, s>>>(a, f, sstart, steps);
    } else {
        (void)cudaGetLastError();  // a refused attribute: the pass stays in global memory
        k_slr_iter_steps<false, kSlrStep * kSlrLanes><<<1, kSlrStep * kSlrLanes, 0, s>>>(a, f, sstart, steps);
    }
    count_launches(1);
}

}  // namespace muto
