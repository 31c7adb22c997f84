// diag.cu -- FP64 diagnostics of a simulation's state (extension).
//
// The reference's only run-time output is an FPS line on the console every
// second (src/main.ts:44-49).  The engine reports conserved quantities
// instead, summed in FP64 over all bodies (original order):
//     M = sum m,  COM = sum m x / M,  P = sum m v,  Lz = sum m (x v_y - y v_x),
//     K = 1/2 sum m |v|^2,
//     W = -G sum_{i<j} m_i m_j / sqrt(|x_i - x_j|^2 + eps_ij^2)
// with the pair softening of the force law in use (Plummer: eps; the
// reference's: eps_ij^2 = epsMult^2 G dt max(m_i, m_j), barnes_hut.wgsl:90-92),
// so that W is the potential whose gradient is the walk's direct-sum force.
//
// moments_kernel: grid-stride FP64 sums, warp shuffles, one FP64 atomic per
// block and quantity.  potential_kernel: the O(N^2) pair sum over unordered
// pairs, tiled through shared memory: a tile's terms m_j / r_ij of a body are
// summed in FP32 (256 at most; rsqrt, relative error ~1e-7 per term) and each
// tile's sum is added into an FP64 accumulator; blocks add m_i-weighted sums
// with one FP64 atomic.  W is for diagnostics, not for every step.
#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "bh.h"
#include "bh_internal.cuh"
#include "packed.cuh"

namespace bh {

constexpr int kDiagThreads = 256;
constexpr int kDiagMoments = 7;  // m, m x, m y, m vx, m vy, Lz, 2K

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

__global__ void __launch_bounds__(kDiagThreads)
moments_kernel(const float* __restrict__ mass, const float2* __restrict__ pos,
               const float2* __restrict__ vel, uint32_t n, double* __restrict__ out) {
    __shared__ double s[kDiagThreads / 32][kDiagMoments];
    double a[kDiagMoments] = {0, 0, 0, 0, 0, 0, 0};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double m = mass[i];
        const float2 x = pos[i], v = vel[i];
        const double px = m * (double)v.x, py = m * (double)v.y;
        a[0] += m;
        a[1] += m * (double)x.x;
        a[2] += m * (double)x.y;
        a[3] += px;
        a[4] += py;
        a[5] += (double)x.x * py - (double)x.y * px;
        a[6] += px * (double)v.x + py * (double)v.y;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kDiagMoments; ++k) {
        const double t = warp_sum_d(a[k]);
        if (lane == 0) s[warp][k] = t;
    }
    __syncthreads();
    if (threadIdx.x < kDiagMoments) {
        double t = 0.0;
        for (int w = 0; w < kDiagThreads / 32; ++w) t += s[w][threadIdx.x];
        atomicAdd(&out[threadIdx.x], t);
    }
}

// Each unordered pair once: a block owns kPotBlock bodies i (kPotPerThread per
// thread, two per packed instruction) and a run of tiles of kPotTile bodies j;
// tiles below its own bodies are another block's, tiles that overlap them take
// the pairs with j > i.  Bound by the reciprocal square roots: 16 a clock and
// SM, one per pair; everything else of a pair takes fewer slots than that.
// A call (B200; every ordered pair with scalar arithmetic, now; the square
// roots alone): 200k bodies 24.0 / 5.0 / 4.3 ms, 800k 429 / 75 / 69 ms.
constexpr int kPotPerThread = 4;
constexpr uint32_t kPotBlock = kDiagThreads * kPotPerThread;
constexpr uint32_t kPotTile = kDiagThreads;

template <bool PLUMMER>
__global__ void __launch_bounds__(kDiagThreads)
potential_kernel(const float* __restrict__ mass, const float2* __restrict__ pos, uint32_t n,
                 float eps2, float eps_coef, uint32_t tiles_per_block, double* __restrict__ out) {
    __shared__ float4 tile[kPotTile][2];  // {x, x, y, y}, {m, m, 0, 0}
    __shared__ double s[kDiagThreads / 32];
    constexpr int NP = kPotPerThread / 2;
    const uint32_t i0 = blockIdx.x * kPotBlock;
    const uint32_t own = i0 / kPotTile;  // first tile with a pair j > i
    const uint32_t tiles = (n + kPotTile - 1) / kPotTile;
    const uint64_t at = (uint64_t)own + (uint64_t)blockIdx.y * tiles_per_block;
    if (at >= tiles) return;  // the shorter runs of later blocks
    const uint32_t t0 = (uint32_t)at;
    const uint32_t t1 = t0 + tiles_per_block < tiles ? t0 + tiles_per_block : tiles;
    f2x X[NP], Y[NP], A[NP];
    float mi[kPotPerThread];
    double acc[kPotPerThread];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        float px[2], py[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t i = i0 + (uint32_t)(2 * q + h) * kDiagThreads + threadIdx.x;
            const bool ok = i < n;
            const float2 p = ok ? pos[i] : make_float2(-kFarAway, -kFarAway);
            px[h] = p.x;
            py[h] = p.y;
            mi[2 * q + h] = ok ? mass[i] : 0.0f;
            acc[2 * q + h] = 0.0;
        }
        X[q] = pk(px[0], px[1]);
        Y[q] = pk(py[0], py[1]);
    }
    const f2x E2 = pk(eps2, eps2);
    for (uint32_t t = t0; t < t1; ++t) {
        __syncthreads();
        {
            const uint32_t j = t * kPotTile + threadIdx.x;
            const float2 p = j < n ? pos[j] : make_float2(kFarAway, kFarAway);
            const float m = j < n ? mass[j] : 0.0f;
            tile[threadIdx.x][0] = make_float4(p.x, p.x, p.y, p.y);
            tile[threadIdx.x][1] = make_float4(m, m, 0.0f, 0.0f);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NP; ++q) A[q] = pk(0.0f, 0.0f);
        const bool overlap = t * kPotTile < i0 + kPotBlock;
        auto pairs = [&](int k, bool after0, bool after1, int q) {
            const float4 o = tile[k][0];
            const f2x M = ld_pair(tile[k][1], 0);
            const f2x dx = sub2(ld_pair(o, 0), X[q]), dy = sub2(ld_pair(o, 1), Y[q]);
            f2x e2 = E2;
            if (!PLUMMER) {
                float m, m1;
                upk(M, m, m1);
                e2 = pk(eps_coef * fmaxf(mi[2 * q], m), eps_coef * fmaxf(mi[2 * q + 1], m));
            }
            const f2x r2 = fma2(dx, dx, fma2(dy, dy, e2));
            float a, b;
            upk(r2, a, b);
            // coincident unsoftened pairs (and ones without a distance) count nothing
            const f2x inv = pk(a > 0.0f && after0 ? rsqrt_ftz(a) : 0.0f,
                               b > 0.0f && after1 ? rsqrt_ftz(b) : 0.0f);
            A[q] = fma2(M, inv, A[q]);
        };
        if (!overlap) {
#pragma unroll 16
            for (int k = 0; k < (int)kPotTile; ++k)
#pragma unroll
                for (int q = 0; q < NP; ++q) pairs(k, true, true, q);
        } else {
#pragma unroll 2
            for (int k = 0; k < (int)kPotTile; ++k) {
                const uint32_t j = t * kPotTile + (uint32_t)k;
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const uint32_t i = i0 + (uint32_t)(2 * q) * kDiagThreads + threadIdx.x;
                    pairs(k, j > i, j > i + kDiagThreads, q);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            float a, b;
            upk(A[q], a, b);
            acc[2 * q] += (double)a;
            acc[2 * q + 1] += (double)b;
        }
    }
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < kPotPerThread; ++k) sum += acc[k] * (double)mi[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double tot = warp_sum_d(sum);
    if (lane == 0) s[warp] = tot;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int w = 0; w < kDiagThreads / 32; ++w) b += s[w];
        atomicAdd(out, b);
    }
}

// FP64 direct-sum acceleration of sampled bodies: block (k, c) adds body
// sample[k]'s pull from the bodies of chunk c.  Consecutive blocks take
// consecutive samples of the same chunk, so the blocks resident together
// read the same ~1M bodies and the chunk is read from DRAM about once.
constexpr uint32_t kDirectChunks = 16;

__global__ void __launch_bounds__(kDiagThreads)
direct_fp64_kernel(const float* __restrict__ mass, const float2* __restrict__ pos, uint32_t n,
                   const uint32_t* __restrict__ sample, int plummer, double eps2, double eps_coef,
                   double* __restrict__ out) {
    __shared__ double s[2][kDiagThreads / 32];
    const uint32_t i = sample[blockIdx.x];
    const uint32_t chunk = (n + gridDim.y - 1) / gridDim.y;
    const uint32_t lo = blockIdx.y * chunk;
    const uint32_t hi = (lo + chunk) < n ? (lo + chunk) : n;
    const float2 pi = pos[i];
    const double xi = pi.x, yi = pi.y, mi = mass[i];
    double ax = 0.0, ay = 0.0;
    for (uint32_t j = lo + threadIdx.x; j < hi; j += kDiagThreads) {
        if (j == i) continue;
        const float2 pj = pos[j];
        const double mj = mass[j];
        const double dx = (double)pj.x - xi, dy = (double)pj.y - yi;
        const double e2 = plummer ? eps2 : eps_coef * fmax(mi, mj);
        const double r2 = dx * dx + dy * dy + e2;
        if (!(r2 > 0.0)) continue;
        const double inv = rsqrt(r2);
        const double f = mj * inv * inv * inv;
        ax += f * dx;
        ay += f * dy;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ax = warp_sum_d(ax);
    ay = warp_sum_d(ay);
    if (lane == 0) {
        s[0][warp] = ax;
        s[1][warp] = ay;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int w = 0; w < kDiagThreads / 32; ++w) t += s[threadIdx.x][w];
        atomicAdd(&out[2 * (size_t)blockIdx.x + threadIdx.x], t);
    }
}

bool sim_body_view(const bh_sim* s, BodyView* out);
void set_global_error(const std::string& msg);

}  // namespace bh

static int dfail(int code, const std::string& msg) {
    bh::set_global_error(msg);
    return code;
}

extern "C" int bh_diagnostics_compute(bh_sim* sim, int with_potential, bh_diagnostics* out) {
    if (!sim || !out) return dfail(BH_ERR_INVALID_ARGUMENT, "bh_diagnostics_compute: null argument");
    bh_config cfg;
    const int st = bh_get_config(sim, &cfg);
    if (st != BH_OK) return st;
    bh::BodyView v;
    bh::sim_body_view(sim, &v);
    cudaError_t e = cudaSetDevice(v.device);
    if (e != cudaSuccess) return dfail(BH_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
    double h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (v.n > 0) {
        // The handle's own 64 bytes: an allocation per call cost more than the
        // sums of 10k bodies (call 549 -> 65 us).
        double* const d = v.diag;
        cudaMemsetAsync(d, 0, sizeof(h), v.stream);
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, v.device);
        uint32_t blocks = (uint32_t)sms * 4u;
        const uint32_t need = (v.n + bh::kDiagThreads - 1) / bh::kDiagThreads;
        if (blocks > need) blocks = need;
        bh::moments_kernel<<<blocks, bh::kDiagThreads, 0, v.stream>>>(v.mass, v.pos, v.vel, v.n, d);
        if (with_potential) {
            const int plummer = cfg.softening == BH_SOFTENING_PLUMMER;
            const float eps2 = cfg.plummer_eps * cfg.plummer_eps;
            // (epsMult sqrt(G dt m))^2, barnes_hut.wgsl:90-92
            const float coef = cfg.epsilon_multiplier * cfg.epsilon_multiplier * cfg.grav_constant *
                               cfg.delta_time;
            const uint32_t own = (v.n + bh::kPotBlock - 1) / bh::kPotBlock;
            const uint32_t tiles = (v.n + bh::kPotTile - 1) / bh::kPotTile;
            // runs of up to 64 tiles, shorter where that leaves fewer than
            // about 16 blocks per SM (half of the grid lies below the diagonal)
            uint64_t run = (uint64_t)own * tiles / (32u * (uint64_t)sms);
            if (run < 1) run = 1;
            if (run > 64) run = 64;
            if (run < tiles / 65535u + 1u) run = tiles / 65535u + 1u;  // grid.y's limit
            const dim3 grid(own, (uint32_t)((tiles + run - 1) / run));
            if (plummer)
                bh::potential_kernel<true><<<grid, bh::kDiagThreads, 0, v.stream>>>(
                    v.mass, v.pos, v.n, eps2, coef, (uint32_t)run, d + 7);
            else
                bh::potential_kernel<false><<<grid, bh::kDiagThreads, 0, v.stream>>>(
                    v.mass, v.pos, v.n, eps2, coef, (uint32_t)run, d + 7);
        }
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, v.stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(v.stream);
        if (e != cudaSuccess) return dfail(BH_ERR_CUDA, std::string("diagnostics: ") + cudaGetErrorString(e));
    }
    out->total_mass = h[0];
    out->com[0] = h[0] > 0.0 ? h[1] / h[0] : 0.0;
    out->com[1] = h[0] > 0.0 ? h[2] / h[0] : 0.0;
    out->momentum[0] = h[3];
    out->momentum[1] = h[4];
    out->angular_momentum = h[5];
    out->kinetic_energy = 0.5 * h[6];
    out->potential_energy = with_potential ? -(double)cfg.grav_constant * h[7] : NAN;
    out->pairs = (with_potential && v.n > 1) ? (uint64_t)v.n * (v.n - 1) / 2 : 0;
    return BH_OK;
}

extern "C" int bh_direct_forces_fp64(bh_sim* sim, const uint32_t* sample, uint32_t count,
                                     double* acc_out) {
    if (!sim || (count && (!sample || !acc_out)))
        return dfail(BH_ERR_INVALID_ARGUMENT, "bh_direct_forces_fp64: null argument");
    if (count > (1u << 20))
        return dfail(BH_ERR_INVALID_ARGUMENT, "bh_direct_forces_fp64: at most 2^20 samples per call");
    bh_config cfg;
    const int st = bh_get_config(sim, &cfg);
    if (st != BH_OK) return st;
    bh::BodyView v;
    bh::sim_body_view(sim, &v);
    for (uint32_t k = 0; k < count; ++k)
        if (sample[k] >= v.n) return dfail(BH_ERR_INVALID_ARGUMENT, "bh_direct_forces_fp64: sample index out of range");
    if (count == 0) return BH_OK;
    cudaError_t e = cudaSetDevice(v.device);
    if (e != cudaSuccess) return dfail(BH_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
    const size_t out_bytes = 2 * sizeof(double) * (size_t)count;
    const size_t idx_off = (out_bytes + 255) & ~(size_t)255;
    unsigned char* d = nullptr;
    e = cudaMallocAsync((void**)&d, idx_off + 4 * (size_t)count, v.stream);
    if (e != cudaSuccess) return dfail(BH_ERR_CUDA, std::string("cudaMallocAsync: ") + cudaGetErrorString(e));
    double* dacc = reinterpret_cast<double*>(d);
    uint32_t* didx = reinterpret_cast<uint32_t*>(d + idx_off);
    e = cudaMemsetAsync(dacc, 0, out_bytes, v.stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(didx, sample, 4 * (size_t)count, cudaMemcpyHostToDevice, v.stream);
    if (e == cudaSuccess) {
        const int plummer = cfg.softening == BH_SOFTENING_PLUMMER;
        const double eps2 = (double)cfg.plummer_eps * (double)cfg.plummer_eps;
        // (epsMult sqrt(G dt m))^2, barnes_hut.wgsl:90-92
        const double coef = (double)cfg.epsilon_multiplier * cfg.epsilon_multiplier *
                            cfg.grav_constant * cfg.delta_time;
        uint32_t chunks = bh::kDirectChunks;
        if (v.n < chunks * bh::kDiagThreads) chunks = 1;
        bh::direct_fp64_kernel<<<dim3(count, chunks), bh::kDiagThreads, 0, v.stream>>>(
            v.mass, v.pos, v.n, didx, plummer, eps2, coef, dacc);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(acc_out, dacc, out_bytes, cudaMemcpyDeviceToHost, v.stream);
    cudaFreeAsync(d, v.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(v.stream);
    if (e != cudaSuccess) return dfail(BH_ERR_CUDA, std::string("direct forces: ") + cudaGetErrorString(e));
    const double G = cfg.grav_constant;
    for (size_t k = 0; k < 2 * (size_t)count; ++k) acc_out[k] *= G;
    return BH_OK;
}
