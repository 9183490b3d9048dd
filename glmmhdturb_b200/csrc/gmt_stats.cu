// gmt_stats.cu -- turbulence statistics on the device: the shell-binned kinetic-energy spectrum, its
// band-limited form with gradient, and the log-density PDF.
//
// E(k) = 1/2 sum_{k-1/2 <= |k'| < k+1/2} |w^(k')|^2 with w = sqrt(rho) v = m / sqrt(rho) and
// w^(k) = N^-3 sum_x w(x) e^{-2 pi i k.x/N}, so that sum_k E(k) is the mean kinetic energy density
// (Parseval).  Only |k_i| <= kmax is needed, so the transform is three separable low-k DFT stages
// (x: kx = 0..kmax, y and z: -kmax..kmax), O(N^3 kmax) work, FP64 accumulation, and fixed-order
// reductions (no atomics: the spectrum is bit-reproducible).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gmt_internal.h"

namespace gmt {

// Twiddles of one axis, tw[k][x] = e^{-2 pi i k x/n} for k = 0..kmax (negative k by conjugation), made on
// the device: k x is reduced modulo n exactly, so sincospi sees an argument in [0, 2).  (On the host
// the cos/sin calls and the three uploads of a 256^3 spectrum took 0.4 ms.)
__global__ void __launch_bounds__(256) twiddle_kernel(int nx, int ny, int nz, int K1, double2* twx, double2* twy,
                                                      double2* twz) {
    const int n = blockIdx.y == 0 ? nx : (blockIdx.y == 1 ? ny : nz);
    double2* t = blockIdx.y == 0 ? twx : (blockIdx.y == 1 ? twy : twz);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K1 * n; i += gridDim.x * blockDim.x) {
        const long long k = i / n, x = i % n;
        double s, c;
        sincospi(2.0 * (double)((k * x) % n) / (double)n, &s, &c);
        t[i] = make_double2(c, -s);
    }
}

// Stage x: A[c][kx][row] = sum_x w_c(x,row) e^{-i 2pi kx x/nx}, row = y + ny z.
// A block takes 32 rows.  Chunks of 32 columns are staged through shared memory, where w = m/sqrt(rho)
// is formed once per cell (one reciprocal root for the three components: the 256^3 statistics call takes 589 us,
// with a root and three divisions 672 us, and E errs by 3.92 and 3.91 x 2^-53 at worst); lane l of every warp
// then owns row l, and warp g accumulates the SX_K wavenumbers g SX_K .. of all three components in
// registers, so a staged value feeds 2 SX_K FMAs and the twiddles are warp-uniform (broadcast) reads.
// 6 (kmax+1) FP64 FMAs and a root per cell; 256^3 FP32, kmax = 8: 208 us, waiting for fixed latencies and for the
// chunk's loads at 10 warps per SM (35.6 KB of shared memory and 64 threads a block).  3.56 ms for one thread per
// (component, kx, row), which read uncoalesced and formed every root 3 (kmax+1) times.
constexpr int SX_K = 5, SX_WARPS = 4, SX_PITCH = 33;
template <class R>
__global__ void __launch_bounds__(32 * SX_WARPS) spec_x_kernel(const CPlanes<R> u, int nx, size_t rows, int K1,
                                                               const double2* __restrict__ tw, double2* __restrict__ A) {
    __shared__ double W[3][32 * SX_PITCH];
    __shared__ double2 T[SX_WARPS * SX_K][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const size_t row0 = (size_t)blockIdx.x * 32;
    const int k0 = (blockIdx.y * nw + warp) * SX_K;          // first wavenumber of this warp
    double re[3][SX_K], im[3][SX_K];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int j = 0; j < SX_K; ++j) re[c][j] = im[c][j] = 0.0;
    for (int xc = 0; xc < nx; xc += 32) {
        const int xw = min(32, nx - xc);
        for (int r0 = warp; r0 < 32; r0 += 4 * nw) {         // a warp reads 32 columns of four rows at a time
            double v[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + q * nw;
                const bool in = r < 32 && lane < xw && row0 + r < rows;
                const size_t g = in ? (row0 + r) * nx + xc + lane : 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) v[q][k] = in ? (double)u.p[k][g] : (k == 0 ? 1.0 : 0.0);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + q * nw, at = r * SX_PITCH + lane;
                if (r >= 32) break;
                const double is = rsqrt(fmax(v[q][0], 1e-300));
                W[0][at] = v[q][1] * is; W[1][at] = v[q][2] * is; W[2][at] = v[q][3] * is;
            }
        }
        for (int i = threadIdx.x; i < nw * SX_K * 32; i += blockDim.x) {
            const int k = blockIdx.y * nw * SX_K + i / 32, x = xc + i % 32;
            T[i / 32][i % 32] = k < K1 && x < nx ? tw[(size_t)k * nx + x] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        if (k0 < K1) {
#pragma unroll 2
            for (int x = 0; x < xw; ++x) {
                const double w0 = W[0][lane * SX_PITCH + x], w1 = W[1][lane * SX_PITCH + x], w2 = W[2][lane * SX_PITCH + x];
#pragma unroll
                for (int j = 0; j < SX_K; ++j) {
                    const double2 e = T[warp * SX_K + j][x];
                    re[0][j] = fma(w0, e.x, re[0][j]); im[0][j] = fma(w0, e.y, im[0][j]);
                    re[1][j] = fma(w1, e.x, re[1][j]); im[1][j] = fma(w1, e.y, im[1][j]);
                    re[2][j] = fma(w2, e.x, re[2][j]); im[2][j] = fma(w2, e.y, im[2][j]);
                }
            }
        }
        __syncthreads();
    }
    const size_t row = row0 + lane;
    if (row >= rows) return;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int j = 0; j < SX_K; ++j)
            if (k0 + j < K1) A[((size_t)c * K1 + k0 + j) * rows + row] = make_double2(re[c][j], im[c][j]);
}

// Stages y and z: O[col][kmax + k] = scale * sum_i I[col][i] e^{-i 2pi k i/n} for k = -kmax..kmax.  One warp
// per (column, group of SYZ_K wavenumbers): the lanes take strided elements, and the four real sums of
// a k >= 0 (re and im of I times cos and sin) give both +k and -k.  The lanes' partial sums are added
// by a fixed shuffle tree.  Output element (col, j) goes to (col / seg) segO + j strO + col % seg, which
// transposes for the next stage.
constexpr int SYZ_K = 3;
__global__ void __launch_bounds__(128) spec_axis_kernel(const double2* __restrict__ I, int n, size_t cols, int kmax,
                                                        const double2* __restrict__ tw, double scale,
                                                        double2* __restrict__ O, size_t seg, size_t segO, size_t strO) {
    const int lane = threadIdx.x & 31, groups = (kmax + SYZ_K) / SYZ_K;
    const size_t job = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (job >= cols * groups) return;
    const size_t col = job / groups;
    const int k0 = (int)(job % groups) * SYZ_K;
    const double2* a = I + col * n;
    double rc[SYZ_K], rs[SYZ_K], ic[SYZ_K], is[SYZ_K];
#pragma unroll
    for (int j = 0; j < SYZ_K; ++j) rc[j] = rs[j] = ic[j] = is[j] = 0.0;
    for (int i = lane; i < n; i += 32) {
        const double2 v = a[i];
#pragma unroll
        for (int j = 0; j < SYZ_K; ++j) {
            if (k0 + j <= kmax) {
                const double2 e = tw[(size_t)(k0 + j) * n + i];
                rc[j] = fma(v.x, e.x, rc[j]); rs[j] = fma(v.x, e.y, rs[j]);
                ic[j] = fma(v.y, e.x, ic[j]); is[j] = fma(v.y, e.y, is[j]);
            }
        }
    }
    double2* o = O + (col / seg) * segO + col % seg;
#pragma unroll
    for (int j = 0; j < SYZ_K; ++j) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            rc[j] += __shfl_xor_sync(0xffffffffu, rc[j], s);
            rs[j] += __shfl_xor_sync(0xffffffffu, rs[j], s);
            ic[j] += __shfl_xor_sync(0xffffffffu, ic[j], s);
            is[j] += __shfl_xor_sync(0xffffffffu, is[j], s);
        }
        const int k = k0 + j;
        if (k <= kmax) {
            // e^{-i th} = (e.x, e.y): v e = (v.x e.x - v.y e.y, v.x e.y + v.y e.x); conjugate for -k
            if (lane == 0) o[(size_t)(kmax + k) * strO] = make_double2((rc[j] - is[j]) * scale, (rs[j] + ic[j]) * scale);
            if (lane == 1 && k > 0) o[(size_t)(kmax - k) * strO] = make_double2((rc[j] + is[j]) * scale, (ic[j] - rs[j]) * scale);
        }
    }
}

__device__ __forceinline__ int shell_of(int kx, int ky, int kz) {
    return (int)floor(sqrt((double)(kx * kx + ky * ky + kz * kz)) + 0.5);
}

// out[b] = 1/2 sum of |C|^2 over the modes whose shell lies in [lo + b step, hi + b step] (the -kx half by
// Hermitian symmetry): one block per shell of a spectrum (lo = hi = 0, step = 1), one block for a band.
// Each thread sums a fixed stride of modes, then a fixed tree.
__global__ void __launch_bounds__(256) spec_shell_kernel(const double2* __restrict__ C, int kmax, int lo, int hi, int step,
                                                         double* out) {
    __shared__ double red[256];
    const int K1 = kmax + 1, K2 = 2 * kmax + 1, modes = K1 * K2 * K2;
    const int s0 = lo + step * (int)blockIdx.x, s1 = hi + step * (int)blockIdx.x;
    double acc = 0.0;
    for (int i = threadIdx.x; i < modes; i += blockDim.x) {
        const int jz = i % K2, jy = (i / K2) % K2, kx = i / (K2 * K2);
        const int sh = shell_of(kx, jy - kmax, jz - kmax);
        if (sh < s0 || sh > s1) continue;
        double p = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double2 v = C[(size_t)c * modes + i];
            p += v.x * v.x + v.y * v.y;
        }
        acc += (kx > 0 ? 1.0 : 0.5) * p;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// scratch of the forward transform: twiddles, A[c][kx][row], B[c][kx][jy][z], C[c][kx][jy][jz]
struct SpecScratch {
    double2 *twx, *twy, *twz, *A, *B, *C, *end;
    static size_t count(int nx, int ny, int nz, int kmax) {   // double2s, in the order of the members
        const size_t K1 = kmax + 1, K2 = 2 * kmax + 1;
        return K1 * ((size_t)nx + ny + nz) + 3 * K1 * ((size_t)ny * nz + K2 * nz + K2 * K2);
    }
    SpecScratch(void* scratch, int nx, int ny, int nz, int kmax) {
        const size_t K1 = kmax + 1, K2 = 2 * kmax + 1;
        twx = static_cast<double2*>(scratch);
        twy = twx + K1 * nx;
        twz = twy + K1 * ny;
        A = twz + K1 * nz;
        B = A + 3 * K1 * (size_t)ny * nz;
        C = B + 3 * K1 * K2 * (size_t)nz;
        end = C + 3 * K1 * K2 * K2;
    }
};

size_t spectrum_scratch_bytes(int nx, int ny, int nz, int kmax) {
    return SpecScratch::count(nx, ny, nz, kmax) * sizeof(double2) + (size_t)(kmax + 1) * sizeof(double) + 256;
}

// C[c][kx][jy][jz] = N^-3 sum_x w_c(x) e^{-i k.x}
template <class R>
static void launch_transform(const CPlanes<R>& u, int nx, int ny, int nz, int kmax, const SpecScratch& S, cudaStream_t s) {
    const int K1 = kmax + 1, K2 = 2 * kmax + 1;
    const size_t rows = (size_t)ny * nz;
    const int top = std::max(nx, std::max(ny, nz));
    twiddle_kernel<<<dim3(std::min((K1 * top + 255) / 256, 148), 3), 256, 0, s>>>(nx, ny, nz, K1, S.twx, S.twy, S.twz);
    const int need = (K1 + SX_K - 1) / SX_K, nw = std::min(need, SX_WARPS);
    spec_x_kernel<R><<<dim3((unsigned)((rows + 31) / 32), (need + nw - 1) / nw), 32 * nw, 0, s>>>(u, nx, rows, K1, S.twx, S.A);
    const int groups = (kmax + SYZ_K) / SYZ_K;
    // y: column (c, kx, z) -> B[c][kx][jy][z]; z: column (c, kx, jy) -> C[c][kx][jy][jz]
    const size_t cy = 3 * (size_t)K1 * nz, cz = 3 * (size_t)K1 * K2;
    spec_axis_kernel<<<(unsigned)((cy * groups + 3) / 4), 128, 0, s>>>(S.A, ny, cy, kmax, S.twy, 1.0, S.B, nz,
                                                                     (size_t)K2 * nz, nz);
    spec_axis_kernel<<<(unsigned)((cz * groups + 3) / 4), 128, 0, s>>>(S.B, nz, cz, kmax, S.twz,
                                                                     1.0 / ((double)nx * ny * nz), S.C, 1, K2, 1);
}

template <class R>
cudaError_t launch_spectrum(const CPlanes<R>& u, int nx, int ny, int nz, int kmax, void* scratch, double* E_host,
                            cudaStream_t s) {
    const SpecScratch S(scratch, nx, ny, nz, kmax);
    double* E = reinterpret_cast<double*>(S.end);
    launch_transform(u, nx, ny, nz, kmax, S, s);
    spec_shell_kernel<<<kmax + 1, 256, 0, s>>>(S.C, kmax, 0, 0, 1, E);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(E_host, E, (size_t)(kmax + 1) * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e;
}

// ---------------------------------------------------------------------------------------------
// Band-limited kinetic-energy loss L = sum_{kmin <= shell <= kmax} E(shell) and its gradient.
// dL/dw(x) = w_S(x)/N^3 with w_S the band-passed field, pulled back through w = m/sqrt(rho).
// ---------------------------------------------------------------------------------------------
// inverse z: G[c][kx][jy][z] = sum_jz mask * C e^{+i kz z}   (tw holds e^{-i k z}, k >= 0)
__global__ void __launch_bounds__(128) band_iz_kernel(const double2* Cc, int nz, int kmax, int kmin, int kmaxb,
                                                      const double2* tw, double2* G) {
    const int K1 = kmax + 1, K2 = 2 * kmax + 1;
    const size_t total = 3 * (size_t)K1 * K2 * nz;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int z = (int)(t % nz);
        const size_t ckxjy = t / nz;
        const int jy = (int)(ckxjy % K2), kx = (int)((ckxjy / K2) % K1);
        double re = 0.0, im = 0.0;
        for (int jz = 0; jz < K2; ++jz) {
            const int kz = jz - kmax;
            int sh = shell_of(kx, jy - kmax, kz);
            if (sh < kmin || sh > kmaxb) continue;
            double2 cv = Cc[ckxjy * K2 + jz];
            double2 e = tw[(size_t)abs(kz) * nz + z];   // e^{-i |kz| z}
            if (kz < 0) e.y = -e.y;                      // e^{-i kz z}; conj = e^{+i kz z}
            re += cv.x * e.x + cv.y * e.y;
            im += cv.y * e.x - cv.x * e.y;
        }
        G[t] = make_double2(re, im);
    }
}

// inverse y: H[c][kx][y + ny z] = sum_jy G[c][kx][jy][z] e^{+i ky y}
__global__ void __launch_bounds__(128) band_iy_kernel(const double2* G, int ny, int nz, int kmax, const double2* tw,
                                                      double2* H) {
    const int K1 = kmax + 1, K2 = 2 * kmax + 1;
    const size_t rows = (size_t)ny * nz;
    const size_t total = 3 * (size_t)K1 * rows;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t row = t % rows;
        const size_t ckx = t / rows;
        const int y = (int)(row % ny), z = (int)(row / ny);
        double re = 0.0, im = 0.0;
        for (int jy = 0; jy < K2; ++jy) {
            const int ky = jy - kmax;
            double2 g = G[(ckx * K2 + jy) * nz + z];
            double2 e = tw[(size_t)abs(ky) * ny + y];
            if (ky < 0) e.y = -e.y;
            re += g.x * e.x + g.y * e.y;
            im += g.y * e.x - g.x * e.y;
        }
        H[t] = make_double2(re, im);
    }
}

// inverse x + chain rule: wS_c = sum_kx wgt Re(H e^{+i kx x}); ubar = dL/du.  The three components of a
// cell share its twiddles.
template <class R>
__global__ void __launch_bounds__(128) band_ix_kernel(const CPlanes<R> u, int nx, int ny, int nz, int kmax,
                                                      const double2* __restrict__ H, const double2* __restrict__ tw,
                                                      double norm, Planes<R> ub) {
    const size_t rows = (size_t)ny * nz;
    const size_t n = rows * nx;
    const int K1 = kmax + 1;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
        const size_t row = n <= 0xffffffffu ? (size_t)((unsigned)c / (unsigned)nx) : c / nx;
        const int x = (int)(c - row * nx);
        double rho = fmax((double)u.p[0][c], 1e-300), isr = 1.0 / sqrt(rho);
        double ws[3] = {0.0, 0.0, 0.0};
        for (int kx = 0; kx < K1; ++kx) {
            const double2 e = tw[(size_t)kx * nx + x];
            const double wgt = kx > 0 ? 2.0 : 1.0;
#pragma unroll
            for (int comp = 0; comp < 3; ++comp) {
                const double2 h = H[((size_t)comp * K1 + kx) * rows + row];
                ws[comp] += wgt * (h.x * e.x + h.y * e.y);   // Re(h * conj(e))
            }
        }
        double rhob = 0.0;
#pragma unroll
        for (int comp = 0; comp < 3; ++comp) {
            double wb = ws[comp] * norm;
            double m = (double)u.p[1 + comp][c];
            ub.p[1 + comp][c] = (R)(wb * isr);
            rhob += -0.5 * wb * m * isr / rho;
        }
        ub.p[0][c] = (R)rhob;
        for (int v = 4; v < 9; ++v) ub.p[v][c] = (R)0;
    }
}

template <class R>
cudaError_t launch_band_loss(const CPlanes<R>& u, int nx, int ny, int nz, int kmin, int kmax, void* scratch, double* L_host,
                             const Planes<R>& ub, cudaStream_t s) {
    const size_t K1 = kmax + 1, K2 = 2 * kmax + 1;
    const SpecScratch S(scratch, nx, ny, nz, kmax);
    double* L = reinterpret_cast<double*>(S.end);
    auto grid = [](size_t total) { return (int)std::min<size_t>((total + 127) / 128, 148 * 32); };
    launch_transform(u, nx, ny, nz, kmax, S, s);
    spec_shell_kernel<<<1, 256, 0, s>>>(S.C, kmax, kmin, kmax, 0, L);
    band_iz_kernel<<<grid(3 * K1 * K2 * nz), 128, 0, s>>>(S.C, nz, kmax, kmin, kmax, S.twz, S.B);
    band_iy_kernel<<<grid(3 * K1 * ny * nz), 128, 0, s>>>(S.B, ny, nz, kmax, S.twy, S.A);
    band_ix_kernel<R><<<grid((size_t)nx * ny * nz), 128, 0, s>>>(u, nx, ny, nz, kmax, S.A, S.twx,
                                                                1.0 / ((double)nx * ny * nz), ub);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(L_host, L, sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e;
}

size_t band_scratch_bytes(int nx, int ny, int nz, int kmax) { return spectrum_scratch_bytes(nx, ny, nz, kmax); }

template cudaError_t launch_band_loss<float>(const CPlanes<float>&, int, int, int, int, int, void*, double*,
                                             const Planes<float>&, cudaStream_t);
template cudaError_t launch_band_loss<double>(const CPlanes<double>&, int, int, int, int, int, void*, double*,
                                              const Planes<double>&, cudaStream_t);

// ---------------------------------------------------------------------------------------------
// Log-density PDF: s = ln(rho / <rho>), its histogram on [smin, smax) and its mean and standard
// deviation sigma_s.  Per-block FP64 partials in a fixed tree order and a one-thread final sum
// (deterministic); the histogram is integer counts.
// ---------------------------------------------------------------------------------------------
constexpr int PDF_BLOCKS = 592, PDF_THREADS = 256;

__device__ __forceinline__ double block_sum256(double v, double* red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int st = PDF_THREADS / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    double r = red[0];
    __syncthreads();
    return r;
}

// f(rho) of every cell of this thread.  QUAD (FP32, 16-byte aligned): one 16-byte load per four cells and
// two in flight per turn; the 4-byte loads of the plain loop left the pass at 1.2 TB/s (256^3: 55 us).
template <bool QUAD, class R, class F> __device__ __forceinline__ void pdf_cells(const R* __restrict__ rho, size_t n, F f) {
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, st = (size_t)gridDim.x * blockDim.x;
    if constexpr (QUAD) {
        const float4* q = reinterpret_cast<const float4*>(rho);
        const size_t nq = n / 4;
#pragma unroll 2
        for (size_t i = i0; i < nq; i += st) {
            const float4 v = __ldg(q + i);
            f((double)v.x); f((double)v.y); f((double)v.z); f((double)v.w);
        }
        for (size_t i = 4 * nq + i0; i < n; i += st) f((double)rho[i]);
    } else {
#pragma unroll 4
        for (size_t i = i0; i < n; i += st) f((double)rho[i]);
    }
}

template <bool QUAD, class R>
__global__ void __launch_bounds__(PDF_THREADS) pdf_mass_kernel(const R* __restrict__ rho, size_t n, double* part) {
    __shared__ double red[PDF_THREADS];
    double m = 0.0;
    pdf_cells<QUAD>(rho, n, [&](double r) { m += r; });
    double t = block_sum256(m, red);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// sum of v[stride b] over the blocks' partials by one block: a fixed stride per thread, then a fixed tree
__device__ __forceinline__ double pdf_sum(const double* v, int stride, double* red) {
    double m = 0.0;
    for (int b = threadIdx.x; b < PDF_BLOCKS; b += PDF_THREADS) m += v[(size_t)stride * b];
    return block_sum256(m, red);
}

// Every block forms <rho> from the mass partials itself (the same value everywhere, the order being
// fixed); one thread adding them between the two passes took 27 us.
template <bool QUAD, class R>
__global__ void __launch_bounds__(PDF_THREADS) pdf_hist_kernel(const R* __restrict__ rho, size_t n, const double* mass,
                                                               int nbins, double smin, double smax, double* part,
                                                               unsigned long long* hist) {
    __shared__ double red[PDF_THREADS];
    extern __shared__ unsigned int hs[];
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) hs[b] = 0u;
    const double mean = pdf_sum(mass, 1, red) / (double)n;   // (its barriers also publish hs)
    const double irm = 1.0 / mean;
    const double idel = (double)nbins / (smax - smin);
    double s1 = 0.0, s2 = 0.0;
    pdf_cells<QUAD>(rho, n, [&](double r) {
        const double sv = log(r * irm);
        s1 += sv;
        s2 += sv * sv;
        const double f = (sv - smin) * idel;
        if (f >= 0.0 && f < (double)nbins) atomicAdd(&hs[(int)f], 1u);
    });
    double t1 = block_sum256(s1, red);
    double t2 = block_sum256(s2, red);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = t1; part[2 * blockIdx.x + 1] = t2; }
    for (int b = threadIdx.x; b < nbins; b += blockDim.x)
        if (hs[b]) atomicAdd(&hist[b], (unsigned long long)hs[b]);
}

__global__ void __launch_bounds__(PDF_THREADS) pdf_final_kernel(const double* mass, const double* part, size_t n,
                                                                double* out) {
    __shared__ double red[PDF_THREADS];
    const double m0 = pdf_sum(mass, 1, red) / (double)n;
    const double s1 = pdf_sum(part, 2, red), s2 = pdf_sum(part + 1, 2, red);
    if (threadIdx.x != 0) return;
    const double m = s1 / (double)n;
    out[0] = m0;
    out[1] = m;
    out[2] = sqrt(fmax(s2 / (double)n - m * m, 0.0));
}

size_t pdf_scratch_bytes(int nbins) { return (size_t)(3 * PDF_BLOCKS + 8) * sizeof(double) + (size_t)nbins * 8; }

template <class R>
cudaError_t launch_density_pdf(const R* rho, size_t n, int nbins, double smin, double smax, void* scratch,
                               double* pdf_host, double* stats_host, cudaStream_t s) {
    double* mass = static_cast<double*>(scratch);          // [PDF_BLOCKS]
    double* part = mass + PDF_BLOCKS;                       // [2 PDF_BLOCKS]
    double* out = part + 2 * PDF_BLOCKS;                    // [mean rho, mean s, sigma_s], then the counts
    unsigned long long* hist = reinterpret_cast<unsigned long long*>(out + 8);
    cudaError_t e = cudaMemsetAsync(hist, 0, (size_t)nbins * 8, s);
    if (e != cudaSuccess) return e;
    const size_t sm = (size_t)nbins * sizeof(unsigned);
    bool quad = false;
    if constexpr (sizeof(R) == 4) {
        if (reinterpret_cast<uintptr_t>(rho) % 16 == 0) {
            quad = true;
            pdf_mass_kernel<true, R><<<PDF_BLOCKS, PDF_THREADS, 0, s>>>(rho, n, mass);
            pdf_hist_kernel<true, R><<<PDF_BLOCKS, PDF_THREADS, sm, s>>>(rho, n, mass, nbins, smin, smax, part, hist);
        }
    }
    if (!quad) {
        pdf_mass_kernel<false, R><<<PDF_BLOCKS, PDF_THREADS, 0, s>>>(rho, n, mass);
        pdf_hist_kernel<false, R><<<PDF_BLOCKS, PDF_THREADS, sm, s>>>(rho, n, mass, nbins, smin, smax, part, hist);
    }
    pdf_final_kernel<<<1, PDF_THREADS, 0, s>>>(mass, part, n, out);
    e = cudaGetLastError();
    std::vector<double> h(8 + (size_t)nbins);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), out, h.size() * 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    for (int i = 0; i < 3; ++i) stats_host[i] = h[i];
    const double ds = (smax - smin) / nbins;
    for (int b = 0; b < nbins; ++b) {
        unsigned long long count;
        std::memcpy(&count, &h[8 + b], 8);
        pdf_host[b] = (double)count / ((double)n * ds);
    }
    return cudaSuccess;
}

template cudaError_t launch_density_pdf<float>(const float*, size_t, int, double, double, void*, double*, double*,
                                               cudaStream_t);
template cudaError_t launch_density_pdf<double>(const double*, size_t, int, double, double, void*, double*, double*,
                                                cudaStream_t);

template cudaError_t launch_spectrum<float>(const CPlanes<float>&, int, int, int, int, void*, double*, cudaStream_t);
template cudaError_t launch_spectrum<double>(const CPlanes<double>&, int, int, int, int, void*, double*, cudaStream_t);

}  // namespace gmt
