// Device-side seeded initial states, written straight into a solve's HBM state.
//
// Same fields as mhd_gpu_solver_b200/workloads.py (the host generator), evaluated on the device:
//   * Fourier state: five spectra C_q[ky][kx] (q = vx, vy, A_z, f1, f2; ky = -K..K, kx = 0..K)
//     drawn on the host; each field is Re(sum_k C_q[k] exp(i 2 pi (kx x + ky y))) at cell centres,
//     B = curl(A_z z^) from the analytic derivatives, v and B scaled to rms 1, f1 and f2 to rms 1,
//     rho = 1 + clip(0.2 f1, +-0.2), p = 1 + clip(0.1 f2, +-0.2), vz = Bz = psi = 0;
//   * four quadrants: per quadrant rho, p, vx, vy, By, with Bx = 0.75;
// then to_conservative (include/mhd/mhd_physics.hpp:41-57). The rms sums are reduced on the device
// in a fixed order.
#pragma once

#include "runtime_types.cuh"
#include "stage_mixed.cuh"

namespace mhdb {

constexpr int kGenThreads = 256;
constexpr int kGenBlocks = 1184; // 8 x 148 SMs

struct GenSpec {
    int kind; // 0 Fourier, 1 four quadrants
    int kmax;
    double gamma;
    double quad[4][5]; // rho, p, vx, vy, by per quadrant (x<.5,y<.5), (x>=.5,y<.5), (x<.5,y>=.5), (x>=.5,y>=.5)
    double x_min, x_max, y_min, y_max;
};

// Raw Fourier fields into the scratch planes: 0 f1, 1 vx, 2 vy, 4 f2, 5 bx, 6 by (unscaled),
// and per-block partial sums of vx^2+vy^2, bx^2+by^2, f1^2, f2^2.
//
// A block takes 256 cells of one row at a time. The sum over ky is the same for all of them, so it
// is done once per item into shared memory, D_q[kx] = sum_ky C_q[ky][kx] exp(i 2 pi ky uy) (and the
// same of i w_y C for A_z's y derivative), and each cell adds KX terms Re(D_q[kx] exp(i 2 pi kx ux))
// with KX sincospi in place of 2 KX KY: FP64-bound, 141 -> 17 us for the mean solve of a batch of
// sides 64-1024 (1.2e5 cells, kmax 8). kx and ky go in chunks, so any kmax fits.
constexpr int kGenChunk = 32;
constexpr int kGenFields = 6; // vx, vy, dA/dy, A (for dA/dx), f1, f2

static __global__ void __launch_bounds__(kGenThreads) gen_fourier_raw(const double2* __restrict__ coef,
                                                              GenSpec s, Geometry g,
                                                              double* __restrict__ scratch,
                                                              double* __restrict__ partial)
{
    const int K = s.kmax;
    const int KX = K + 1, KY = 2 * K + 1, NC = KX * KY;
    const double wx = 2.0 * M_PI / (s.x_max - s.x_min), wy = 2.0 * M_PI / (s.y_max - s.y_min);
    __shared__ double2 ey[kGenChunk];
    __shared__ double2 D[kGenChunk][kGenFields];
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const int tiles_x = (g.nx + kGenThreads - 1) / kGenThreads;
    const long long items = static_cast<long long>(tiles_x) * g.ny;
    for (long long it = blockIdx.x; it < items; it += gridDim.x) {
        const int y = static_cast<int>(it / tiles_x);
        const int x = static_cast<int>(it % tiles_x) * kGenThreads + static_cast<int>(threadIdx.x);
        const double ux = (x + 0.5) / g.nx, uy = (y + 0.5) / g.ny; // (x - x_min)/lx
        double v[kGenFields] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int kx0 = 0; kx0 < KX; kx0 += kGenChunk) {
            const int nkx = min(kGenChunk, KX - kx0);
            // D of this chunk: one (kx, field) per thread
            const int dk = threadIdx.x % kGenChunk, dq = threadIdx.x / kGenChunk;
            const bool dwork = dq < kGenFields && dk < nkx;
            double dr = 0.0, di = 0.0;
            for (int iy0 = 0; iy0 < KY; iy0 += kGenChunk) {
                const int nky = min(kGenChunk, KY - iy0);
                __syncthreads(); // the previous chunk's ey and D have been read
                if (static_cast<int>(threadIdx.x) < nky) {
                    double sy, cy;
                    sincospi(2.0 * (iy0 + static_cast<int>(threadIdx.x) - K) * uy, &sy, &cy);
                    ey[threadIdx.x] = make_double2(cy, sy);
                }
                __syncthreads();
                if (dwork) {
                    // spectra: 0 vx, 1 vy, 2 A_z, 3 f1, 4 f2
                    const int spec = dq < 2 ? dq : (dq < 4 ? 2 : dq - 1);
                    for (int j = 0; j < nky; ++j) {
                        const double2 c = coef[spec * NC + (iy0 + j) * KX + kx0 + dk];
                        const double er = ey[j].x, ei = ey[j].y;
                        const double pr = c.x * er - c.y * ei, pi = c.x * ei + c.y * er;
                        if (dq == 2) { // times i w_y ky
                            const double w = wy * (iy0 + j - K);
                            dr -= w * pi;
                            di += w * pr;
                        } else {
                            dr += pr;
                            di += pi;
                        }
                    }
                }
            }
            if (dwork) {
                if (dq == 3) { // times -i w_x kx: By = -dA/dx
                    const double w = wx * (kx0 + dk);
                    D[dk][dq] = make_double2(w * di, -w * dr);
                } else {
                    D[dk][dq] = make_double2(dr, di);
                }
            }
            __syncthreads();
            if (x < g.nx) {
                for (int k = 0; k < nkx; ++k) {
                    double sx, cx;
                    sincospi(2.0 * (kx0 + k) * ux, &sx, &cx);
#pragma unroll
                    for (int q = 0; q < kGenFields; ++q) {
                        v[q] += D[k][q].x * cx - D[k][q].y * sx;
                    }
                }
            }
        }
        if (x < g.nx) {
            const size_t o = static_cast<size_t>(y) * g.pitch + x;
            scratch[0 * g.plane + o] = v[4];
            scratch[1 * g.plane + o] = v[0];
            scratch[2 * g.plane + o] = v[1];
            scratch[4 * g.plane + o] = v[5];
            scratch[5 * g.plane + o] = v[2];
            scratch[6 * g.plane + o] = v[3];
            acc[0] += v[0] * v[0] + v[1] * v[1];
            acc[1] += v[2] * v[2] + v[3] * v[3];
            acc[2] += v[4] * v[4];
            acc[3] += v[5] * v[5];
        }
    }
    __shared__ double sh[4][kGenThreads];
    for (int q = 0; q < 4; ++q) {
        sh[q][threadIdx.x] = acc[q];
    }
    __syncthreads();
    for (int st = kGenThreads / 2; st > 0; st >>= 1) {
        if (static_cast<int>(threadIdx.x) < st) {
            for (int q = 0; q < 4; ++q) {
                sh[q][threadIdx.x] += sh[q][threadIdx.x + st];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 4) {
        partial[threadIdx.x * gridDim.x + blockIdx.x] = sh[threadIdx.x][0];
    }
}

template <class Store>
__global__ void __launch_bounds__(kGenThreads) gen_finish(Store store, GenSpec s, Geometry g,
                                                         const double* __restrict__ scratch,
                                                         const double* __restrict__ partial,
                                                         int nblocks)
{
    // scale factors from the block partials: warp q sums the q-th, in a fixed order
    __shared__ double sum[4];
    if (threadIdx.x < 128) {
        const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
        double v = 0.0;
        if (s.kind == 0) {
            for (int b = lane; b < nblocks; b += 32) {
                v += partial[q * nblocks + b];
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (lane == 0) {
            sum[q] = v;
        }
    }
    __syncthreads();
    const double ncell = static_cast<double>(g.nx) * g.ny;
    const double vs = 1.0 / sqrt(sum[0] / ncell), bs = 1.0 / sqrt(sum[1] / ncell);
    const double f1s = sqrt(sum[2] / ncell), f2s = sqrt(sum[3] / ncell);
    const long long n = static_cast<long long>(g.nx) * g.ny;
    for (long long c = blockIdx.x * static_cast<long long>(kGenThreads) + threadIdx.x; c < n;
         c += static_cast<long long>(gridDim.x) * kGenThreads) {
        const int x = static_cast<int>(c % g.nx), y = static_cast<int>(c / g.nx);
        const size_t o = static_cast<size_t>(y) * g.pitch + x;
        double rho, p, vx, vy, bx, by;
        if (s.kind == 0) {
            vx = scratch[1 * g.plane + o] * vs;
            vy = scratch[2 * g.plane + o] * vs;
            bx = scratch[5 * g.plane + o] * bs;
            by = scratch[6 * g.plane + o] * bs;
            const double f1 = scratch[0 * g.plane + o] / f1s;
            const double f2 = scratch[4 * g.plane + o] / f2s;
            rho = 1.0 + fmin(fmax(0.2 * f1, -0.2), 0.2);
            p = 1.0 + fmin(fmax(0.1 * f2, -0.2), 0.2);
        } else {
            const double xc = s.x_min + (x + 0.5) * ((s.x_max - s.x_min) / g.nx);
            const double yc = s.y_min + (y + 0.5) * ((s.y_max - s.y_min) / g.ny);
            const int qd = (xc < 0.5 ? 0 : 1) + (yc < 0.5 ? 0 : 2);
            rho = s.quad[qd][0];
            p = s.quad[qd][1];
            vx = s.quad[qd][2];
            vy = s.quad[qd][3];
            by = s.quad[qd][4];
            bx = 0.75;
        }
        const double e_kin = 0.5 * rho * (vx * vx + vy * vy);
        const double e_mag = 0.5 * (bx * bx + by * by);
        const double u[9] = {rho, rho * vx, rho * vy, 0.0, p / (s.gamma - 1.0) + e_kin + e_mag,
                             bx, by, 0.0, 0.0};
        store(o, u);
    }
}

struct StoreF64 {
    double* u;
    size_t plane;
    __device__ void operator()(size_t o, const double* v) const
    {
        for (int c = 0; c < 9; ++c) {
            u[c * plane + o] = v[c];
        }
    }
};

struct StoreMx {
    MixedState u;
    size_t plane;
    __device__ void operator()(size_t o, const double* v) const
    {
        for (int c = 0; c < 9; ++c) {
            split_store(u, c * plane + o, v[c]);
        }
    }
};

} // namespace mhdb

namespace mhdb {

// Host side: generate an initial state into `store` using `scratch` (9 double planes of the
// solve's geometry, e.g. its stage buffer). The spectra and the rms partials go into scratch's last
// two planes, which the raw fields leave free (stream-ordered allocations in their place made
// admitting a solve wait 2-6 ms for the driver: the default pool gives its memory back at every
// synchronisation); only a grid too small to hold them allocates two stream-ordered buffers.
template <class Store>
inline cudaError_t launch_generate(cudaStream_t st, const GenSpec& spec, const double* coef_host,
                                   const Geometry& g, double* scratch, Store store)
{
    if (spec.kind != 0) {
        gen_finish<<<kGenBlocks, kGenThreads, 0, st>>>(store, spec, g, scratch, nullptr, 0);
        return cudaGetLastError();
    }
    const int nblocks = kGenBlocks;
    const size_t nc = static_cast<size_t>(5) * (2 * spec.kmax + 1) * (spec.kmax + 1);
    const bool fits = 2 * nc + 4 * nblocks <= 2 * g.plane;
    double2* coef = reinterpret_cast<double2*>(scratch + 7 * g.plane); // plane: a multiple of 32
    double* partial = scratch + 7 * g.plane + 2 * nc;
    cudaError_t e = cudaSuccess;
    if (!fits) {
        if ((e = cudaMallocAsync(reinterpret_cast<void**>(&coef), nc * sizeof(double2), st)) != cudaSuccess) {
            return e;
        }
        if ((e = cudaMallocAsync(reinterpret_cast<void**>(&partial), 4 * nblocks * sizeof(double), st)) != cudaSuccess) {
            cudaFreeAsync(coef, st);
            return e;
        }
    }
    e = cudaMemcpyAsync(coef, coef_host, nc * sizeof(double2), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        gen_fourier_raw<<<nblocks, kGenThreads, 0, st>>>(coef, spec, g, scratch, partial);
        gen_finish<<<nblocks, kGenThreads, 0, st>>>(store, spec, g, scratch, partial, nblocks);
        e = cudaGetLastError();
    }
    if (!fits) {
        cudaFreeAsync(coef, st);
        cudaFreeAsync(partial, st);
    }
    return e;
}

} // namespace mhdb
