// Reciprocal-space PME on caller-owned device buffers that allocates nothing:
// every intermediate (fixed-point charge grid, half spectrum, real grid,
// influence function, per-axis tables, FFT twiddles, energy word) lives in one file-scope device array of fixed size, g_pme_scratch.
//
// The arithmetic is the engine's mixed-precision PME step (k_pme.cu spread
// and gather, k_fft.cu transforms, the influence function of nxm_engine.cu),
// all computed on the device so that one call is a sequence of kernel
// launches on the caller's stream and nothing else: no cudaMalloc, cudaFree,
// host<->device copy or library call that allocates.  It has no counterpart
// in the reference, whose PME (core/baseline/src/Forces/NonbondedForce.cpp
// :51-461) allocates its grids per evaluation.
//
// Limits: each grid axis K in [5, 64] with K = 2^a 3^b 5^c; any atom count.
// Scratch: about 3.7 MB of device memory per device, for the lifetime of
// the library.
//
// Set-up: the first call on a device (the device current at the call) looks
// up the array's device address with cudaGetSymbolAddress, once, and keeps
// it; that lookup may load the module, so the first call on each device
// should come before any stream capture.  The kept address belongs to the
// device's primary context of that time: after cudaDeviceReset (which
// destroys it) the library must be unloaded and loaded again before the
// next call.
//
// Sharing: every call on a device uses the same array, which keeps the
// previous call's contents.  Each call clears what must start at zero (the
// charge-grid accumulator and the energy word) and rewrites everything else
// before reading it.  Calls whose work overlaps on the GPU (two streams, or
// two host threads) race on the array and give wrong results; serialise them.
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <string>

#include "../../include/nxm.h"
#include "nxm_chain.cuh"
#include "nxm_fft.h"
#include "nxm_spread.cuh"
#include "nxm_view.h"

namespace nxm {
int fail(int code, const std::string &msg);
}

namespace {

using namespace nxm;

constexpr int kStaticMaxK = 64;
constexpr int kStaticMaxKh = kStaticMaxK / 2 + 1;
constexpr int kZLines = 16;  // real lines per block in the z passes
constexpr int kCols = 8;     // columns per block in the y and x passes
constexpr size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// byte offsets of the regions of g_pme_scratch
constexpr size_t kOffE = 0;                                                   // long long[E_SLOTS]
constexpr size_t kOffTw = kOffE + align256(sizeof(long long) * E_SLOTS);      // float2[3][K]
constexpr size_t kOffAxis = kOffTw + align256(sizeof(float2) * 3 * kStaticMaxK);  // double2[3][K]
constexpr size_t kOffAcc = kOffAxis + align256(sizeof(double2) * 3 * kStaticMaxK);
constexpr size_t kGridPts = (size_t)kStaticMaxK * kStaticMaxK * kStaticMaxK;
constexpr size_t kSpecPts = (size_t)kStaticMaxK * kStaticMaxK * kStaticMaxKh;
constexpr size_t kOffReal = kOffAcc + align256(sizeof(int) * kGridPts);
constexpr size_t kOffCplx = kOffReal + align256(sizeof(float) * kGridPts);
constexpr size_t kOffEterm = kOffCplx + align256(sizeof(float2) * kSpecPts);
constexpr size_t kScratchBytes = kOffEterm + align256(sizeof(float) * kSpecPts);

__device__ __align__(256) unsigned char g_pme_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
unsigned char *g_scratch_ptr[kMaxDevices] = {};

struct Geometry {
    int K[3];
    int Kh;
    double L[3], invL[3];
    double alpha;
};

template <typename T>
__device__ __forceinline__ T *region(unsigned char *base, size_t off) {
    return reinterpret_cast<T *>(base + off);
}

// Grid base index and fraction of one coordinate (NonbondedForce.cpp:51-71:
// the grid is anchored at the origin).
__device__ __forceinline__ void grid_coord(double p, double invL, int K, int &idx, float &fr) {
    double t = p * invL;
    t = (t - floor(t)) * K;
    int ti = (int)t;
    fr = (float)(t - ti);
    idx = ti > 0 ? ti % K : 0;  // (not finite: the least integer)
}

// |b(k)|^2 of one axis: the order-5 spline's values at the integers are
// 1/24, 11/24, 11/24, 1/24, so with c = cos(2 pi k / K) the sum
// |1/24 (z + z^4) + 11/24 (z^2 + z^3)|^2 is 2 (1 + c) (11/24 + (2c - 1)/24)^2
// (NonbondedForce.cpp:75-142 sums sines and cosines: ten times the FP64 work).
__device__ __forceinline__ double modulus2(int k, int K) {
    const double c = cospi(2.0 * (double)k / (double)K);
    const double t = (10.0 + 2.0 * c) * (1.0 / 24.0);
    return 2.0 * (1.0 + c) * t * t;
}

// ---- set-up, blocks of one warp's worth of FP64 work each (the pipe is
// narrow): the first kAxisBlocks blocks make the per-axis tables -- twiddles,
// and (m_d^2, exp(-pi^2 m_d^2 / alpha^2) / |b|^2) -- one entry per lane, with
// the neighbour average for |b|^2 below 1e-7; the others clear the
// accumulator and the energy words.  The axis tables replace an exponential
// and a modulus sum per spectrum element and a serial block of sines and
// cosines: 24,000 atoms on 64^3, the whole entry 130 -> 77 us.
constexpr int kAxisBlocks = 3 * kStaticMaxK / 32;

__global__ void __launch_bounds__(256) k_noalloc_setup(unsigned char *scr, Geometry g) {
    chain_link();
    if (blockIdx.x >= kAxisBlocks) {
        int4 *acc = region<int4>(scr, kOffAcc);
        const int n = (g.K[0] * g.K[1] * g.K[2] + 3) / 4;  // (the region holds whole int4)
        const int t0 = (blockIdx.x - kAxisBlocks) * blockDim.x + threadIdx.x, nt = (gridDim.x - kAxisBlocks) * blockDim.x;
        for (int i = t0; i < n; i += nt) acc[i] = make_int4(0, 0, 0, 0);
        if (t0 < E_SLOTS) region<long long>(scr, kOffE)[t0] = 0;
        return;
    }
    if (threadIdx.x >= 32) return;
    const int d = blockIdx.x / (kStaticMaxK / 32), k = (blockIdx.x % (kStaticMaxK / 32)) * 32 + threadIdx.x;
    const int K = g.K[d];
    if (k >= K) return;
    {
        double s, c;
        sincospi(-2.0 * (double)k / (double)K, &s, &c);
        region<float2>(scr, kOffTw)[(d > 0 ? g.K[0] : 0) + (d > 1 ? g.K[1] : 0) + k] = make_float2((float)c, (float)s);
    }
    double mod = modulus2(k, K);
    if (mod < 1e-7) mod = (modulus2((k - 1 + K) % K, K) + modulus2((k + 1) % K, K)) / 2.0;
    const double mh = (k < (K + 1) / 2 ? k : k - K) * g.invL[d];
    const double m2 = mh * mh;
    region<double2>(scr, kOffAxis)[d * kStaticMaxK + k] =
        make_double2(m2, exp(-(kPi * kPi / (g.alpha * g.alpha)) * m2) / mod);
}

// 1 / x to 2^-50 from the FP32 reciprocal and two Newton steps (an FP64
// division takes three times the FP64 instructions).
__device__ __forceinline__ double reciprocal(double x) {
    if (!(x > 1e-30 && x < 1e30)) return 1.0 / x;
    double r = (double)fast_rcp((float)x);
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

// ---- spread (the first nspread blocks; a warp takes kAtoms atoms one after
// the other, as the engine's k_spread_warp: int32 fixed point, 2^-24 e, the
// grid word the FFT's first pass reads) and, in the blocks behind, the
// influence function on the half spectrum (NonbondedForce.cpp:323-388), which
// needs the axis tables only: one launch for the two.
constexpr int kAtoms = 8, kSpreadBlockWarps = 4;

__global__ void __launch_bounds__(kSpreadBlockWarps * 32) k_noalloc_spread(unsigned char *scr, Geometry g,
                                                                           const double *xyz, const double *charge,
                                                                           int n, int nspread) {
    chain_link();
    if ((int)blockIdx.x >= nspread) {
        const double2 *ax = region<double2>(scr, kOffAxis), *ay = ax + kStaticMaxK, *az = ay + kStaticMaxK;
        float *et = region<float>(scr, kOffEterm);
        const int K1 = g.K[1], Kh = g.Kh, total = g.K[0] * K1 * Kh;
        const double f = kOne4PiEps0 / (kPi * g.L[0] * g.L[1] * g.L[2]);
        for (int i = (blockIdx.x - nspread) * blockDim.x + threadIdx.x; i < total;
             i += (gridDim.x - nspread) * blockDim.x) {
            const int r = i / Kh, kz = i - r * Kh, kx = r / K1, ky = r - kx * K1;
            const double2 x = ax[kx], y = ay[ky], z = az[kz];
            et[i] = i == 0 ? 0.f : (float)(f * x.y * y.y * z.y * reciprocal(x.x + y.x + z.x));
        }
        return;
    }
    __shared__ float s_w[kSpreadBlockWarps][kAtoms][16];  // wx[5] wy[5] wz[5] q
    __shared__ int s_i[kSpreadBlockWarps][kAtoms][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = (blockIdx.x * kSpreadBlockWarps + warp) * kAtoms;
    // lane 3 a + d prepares axis d of atom a
    if (lane < 3 * kAtoms && first + lane / 3 < n) {
        const int a = lane / 3, d = lane - 3 * a;
        const size_t i = (size_t)first + a;
        int idx;
        float fr, th[5], dth[5];
        grid_coord(xyz[3 * i + d], g.invL[d], g.K[d], idx, fr);
        bspline5<float>(fr, th, dth);
        s_i[warp][a][d] = idx;
#pragma unroll
        for (int k = 0; k < 5; ++k) s_w[warp][a][5 * d + k] = th[k];
        if (d == 0) s_w[warp][a][15] = (float)charge[i];
    }
    __syncwarp();
    int *acc = region<int>(scr, kOffAcc);
    for (int a = 0; a < min(kAtoms, n - first); ++a)
        spread_points(s_w[warp][a], s_i[warp][a], g.K[0], g.K[1], g.K[2], acc, lane);
}

// ---- gather: one thread per atom, the stencil row by row (the z sums first,
// then the row's x/y weights); writes the force (kJ/mol/nm) and, from thread
// 0, the reciprocal energy.
constexpr int kGatherThreads = 64;

__global__ void __launch_bounds__(kGatherThreads) k_noalloc_gather(unsigned char *scr, Geometry g, const double *xyz,
                                                                   const double *charge, int n, double *force,
                                                                   double *energy) {
    chain_link();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *energy = (double)region<long long>(scr, kOffE)[E_RECIP] * kEnergyUnscale;
    if (i >= n) return;
    int idx[3];
    float fr[3], th[3][5], dth[3][5];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        grid_coord(xyz[3 * (size_t)i + d], g.invL[d], g.K[d], idx[d], fr[d]);
        bspline5<float>(fr[d], th[d], dth[d]);
    }
    const float *grid = region<float>(scr, kOffReal);
    const int K0 = g.K[0], K1 = g.K[1], K2 = g.K[2];
    int zo[5];
#pragma unroll
    for (int iz = 0; iz < 5; ++iz) {
        const int zi = idx[2] + iz;
        zo[iz] = zi >= K2 ? zi - K2 : zi;
    }
    float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll
    for (int ix = 0; ix < 5; ++ix) {
        int xi = idx[0] + ix;
        xi -= xi >= K0 ? K0 : 0;
#pragma unroll
        for (int iy = 0; iy < 5; ++iy) {
            int yi = idx[1] + iy;
            yi -= yi >= K1 ? K1 : 0;
            const float *row = grid + (xi * K1 + yi) * K2;
            float sz = 0.f, sdz = 0.f;
#pragma unroll
            for (int iz = 0; iz < 5; ++iz) {
                const float gv = row[zo[iz]];
                sz = fmaf(th[2][iz], gv, sz);
                sdz = fmaf(dth[2][iz], gv, sdz);
            }
            fx = fmaf(dth[0][ix] * th[1][iy], sz, fx);
            fy = fmaf(th[0][ix] * dth[1][iy], sz, fy);
            fz = fmaf(th[0][ix] * th[1][iy], sdz, fz);
        }
    }
    float q = (float)charge[i];
    force[3 * (size_t)i] = (double)(-(q * (fx * (float)(K0 * g.invL[0]))));
    force[3 * (size_t)i + 1] = (double)(-(q * (fy * (float)(K1 * g.invL[1]))));
    force[3 * (size_t)i + 2] = (double)(-(q * (fz * (float)(K2 * g.invL[2]))));
}

bool smooth235(int n) {
    if (n < 1) return false;
    for (int p : {2, 3, 5})
        while (n % p == 0) n /= p;
    return n == 1;
}

// Device address of g_pme_scratch on the current device, looked up once.
int scratch_for_current_device(unsigned char **out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(NXM_ERR_CUDA, std::string("nxm_pme_reciprocal_noalloc: cudaGetDevice: ") +
                                                        cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(NXM_ERR_CUDA, "nxm_pme_reciprocal_noalloc: device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (!g_scratch_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_pme_scratch);
        if (e != cudaSuccess || !p)
            return fail(NXM_ERR_CUDA, std::string("nxm_pme_reciprocal_noalloc: cudaGetSymbolAddress: ") +
                                          cudaGetErrorString(e));
        g_scratch_ptr[dev] = static_cast<unsigned char *>(p);
    }
    *out = g_scratch_ptr[dev];
    return NXM_OK;
}

}  // namespace

extern "C" int nxm_pme_reciprocal_noalloc(const double *xyz, const double *charge, int32_t n_atoms,
                                          const double box_lb[3], const double box_ub[3],
                                          const int32_t grid[3], double alpha, double *force,
                                          double *energy, void *stream) {
    const char *fn = "nxm_pme_reciprocal_noalloc: ";
    if (n_atoms < 0 || !box_lb || !box_ub || !grid || !energy || (n_atoms > 0 && (!xyz || !charge || !force)))
        return fail(NXM_ERR_INVALID, std::string(fn) + "null argument or negative atom count");
    if (!(alpha > 0) || !(alpha < 1e300)) return fail(NXM_ERR_INVALID, std::string(fn) + "alpha must be positive");
    Geometry g{};
    for (int d = 0; d < 3; ++d) {
        if (grid[d] > kStaticMaxK) {
            char msg[160];
            std::snprintf(msg, sizeof msg, "%sgrid %dx%dx%d exceeds the static scratch limit of %d points per axis",
                          fn, grid[0], grid[1], grid[2], kStaticMaxK);
            return fail(NXM_ERR_CAPACITY, msg);
        }
        if (grid[d] < 5 || !smooth235(grid[d]))
            return fail(NXM_ERR_INVALID, std::string(fn) + "grid sizes must be 2^a 3^b 5^c and >= 5");
        g.K[d] = grid[d];
        g.L[d] = box_ub[d] - box_lb[d];
        if (g.L[d] < 0) g.L[d] = -g.L[d];
        if (!(g.L[d] > 0) || !(g.L[d] < 1e300)) return fail(NXM_ERR_INVALID, std::string(fn) + "empty box");
        g.invL[d] = 1 / g.L[d];
    }
    g.Kh = g.K[2] / 2 + 1;
    g.alpha = alpha;
    unsigned char *scr = nullptr;
    int rc = scratch_for_current_device(&scr);
    if (rc != NXM_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    FftSysDev F{};
    int tw = 0;
    for (int d = 0; d < 3; ++d) {
        F.K[d] = g.K[d];
        F.tw[d] = tw;
        tw += g.K[d];
        fft_passes(g.K[d], F.ax[d]);
    }
    fft_passes_reversed(g.K[0], F.ax[0], F.axi);
    F.Kh = g.Kh;
    FftPlan plan;  // geometry only; every pointer is into g_pme_scratch
    plan.S = 1;
    plan.zlines = kZLines;
    plan.cols = kCols;
    plan.nz = (g.K[0] * g.K[1] + kZLines - 1) / kZLines;
    plan.ny = (g.K[0] * g.Kh + kCols - 1) / kCols;
    plan.nx = (g.K[1] * g.Kh + kCols - 1) / kCols;
    plan.hsys.assign(1, F);
    plan.zthreads = fft_line_threads(plan.hsys, 2, kZLines / 2);
    plan.cthreads = std::max(fft_line_threads(plan.hsys, 0, kCols), fft_line_threads(plan.hsys, 1, kCols));
    plan.kmax = std::max(g.K[0], std::max(g.K[1], g.K[2]));
    // line path (plan.plane = 0); at most 64 points per axis keeps every
    // block under the 48 KB that needs no shared-memory attribute
    plan.smem_z = fft_line_smem(kZLines / 2, plan.kmax, sizeof(float2));
    plan.smem_y = fft_line_smem(kCols, plan.kmax, sizeof(float2));
    plan.smem_x = plan.smem_y;
    DevView v{};
    v.N = n_atoms;
    v.S = 1;
    v.mixed = 1;
    v.force_mask = NXM_FORCE_NONBONDED;
    v.grid_acc = scr + kOffAcc;
    v.grid_real = scr + kOffReal;
    v.grid_cplx = scr + kOffCplx;
    v.eterm = scr + kOffEterm;
    v.twiddle = scr + kOffTw;
    v.E = reinterpret_cast<long long *>(scr + kOffE);
    v.total_grid = (long long)g.K[0] * g.K[1] * g.K[2];
    v.total_cgrid = (long long)g.K[0] * g.K[1] * g.Kh;

    // an error already pending on this thread belongs to the caller's earlier
    // work: report it and leave it pending rather than clear it
    cudaError_t pending = cudaPeekAtLastError();
    if (pending != cudaSuccess)
        return fail(NXM_ERR_CUDA, std::string(fn) + "a CUDA error was already pending: " +
                                      cudaGetErrorString(pending));
    k_noalloc_setup<<<kAxisBlocks + kSMs, 256, 0, st>>>(scr, g);
    const int nspread = (n_atoms + kSpreadBlockWarps * kAtoms - 1) / (kSpreadBlockWarps * kAtoms);
    const int neterm = (int)std::min<long long>((v.total_cgrid + kSpreadBlockWarps * 32 - 1) / (kSpreadBlockWarps * 32), 4 * kSMs);
    // (the first kernel is an ordinary launch: it follows whatever the caller
    // put on the stream)
    plan.chained = true;
    launch_link(true, k_noalloc_spread, nspread + neterm, kSpreadBlockWarps * 32, 0, st, scr, g, xyz, charge, n_atoms,
                nspread);
    launch_fft_convolve(v, plan, 1, st);
    launch_link(true, k_noalloc_gather, std::max(1, (n_atoms + kGatherThreads - 1) / kGatherThreads), kGatherThreads, 0,
                st, scr, g, xyz, charge, n_atoms, force, energy);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(NXM_ERR_CUDA, std::string(fn) + "launch failed: " + cudaGetErrorString(e));
    return NXM_OK;
}
