// gmt_passes.cuh -- the unsplit GLM step as three passes over z slabs, for FP64.
//
//   prim    Q  = primitives of the slab's planes and two ghost planes either side
//   recon   MH = the MUSCL-Hancock predictor of every cell (and PPM's "use parabola" flag)
//   flux    interface states mh +- s_d from Q and MH, one Riemann solve per face, update, floor,
//           psi damping, forcing kick, CFL maxima
//
// Why: the fused tile march (gmt_unsplit.cuh) carries 36 values of the column and the whole
// reconstruction of a cell through the Riemann solves.  In FP32 that fits 128 registers; in FP64 it
// takes 255 registers with 360 bytes of spills, 214 KB of shared memory and so 8 warps per SM, whose
// dependent FP64 chains leave the FP64 pipes three quarters idle.  Cut at the predictor, each pass has
// a small working set and enough warps in flight, for 18 planes of scratch written and read once
// (slab-sized, so it is bounded and, for small boxes, stays in L2).  Every value is formed by the
// expressions of the tile march in the same order, so the result is the same bit for bit.
// MC + HLLD with forcing and CFL, tile march -> passes: 32^3 133 -> 87 us, 64^3 251 -> 141 us, 128^3 1.79 -> 1.02
// ms, 192^3 5.83 -> 3.25 ms, 256^3 13.7 -> 8.0 ms, 512^3 110 -> 64.7 ms.  At 128^3 (profiled) the primitives take 44 us, at
// 73 % of the memory's rate; the predictor 147 us at 12 warps per SM (MC's 168 registers), the busiest pipe 62 %
// of its time; the fluxes 778 us at 16 warps per SM (128 registers, 56 bytes spilled; PPM 32 to 96), waiting for
// fixed latencies, for one another at the barriers (24 threads solve a fourth face) and for instructions.
#pragma once
#include "gmt_unsplit.cuh"

namespace gmt {

template <class R> struct PassArgs {
    UnsplitArgs<R> A;
    R* q;                // [9][S + 4][ny][nx]: planes zs - 2 .. zs + S + 1
    R* mh;               // [9][S + 2][ny][nx]: planes zs - 1 .. zs + S
    unsigned char* up;   // PPM only: [S + 2][ny][nx]
    int zs, S, lz;       // slab [zs, zs + S); planes per block of the flux pass
};

// primitives: one thread per cell, plane blockIdx.y of the slab's S + 4
template <class R> __global__ void __launch_bounds__(256) pass_prim_kernel(const PassArgs<R> P) {
    const UnsplitArgs<R>& A = P.A;
    const size_t nxy = (size_t)A.nx * A.ny, qn = nxy * (P.S + 4);
    const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nxy) return;
    const int k = blockIdx.y;
    const size_t g = c + nxy * wrapi(P.zs - 2 + k, A.nz);
    Q9<R> u;
#pragma unroll
    for (int v = 0; v < 9; ++v) u.v[v] = __ldg(A.u.p[v] + g);
    u = cons2prim(u, A.K.gamma, A.K.smallr, A.K.pfl);
#pragma unroll
    for (int v = 0; v < 9; ++v) P.q[v * qn + k * nxy + c] = u.v[v];
}

// half slope without the multiplications by 2: scalings by powers of two are exact, so this is
// half_slope1 up to the sign of a zero slope, which no sum sees
template <bool MM, class R> __device__ __forceinline__ R pass_slope(R dl, R dr) {
    if constexpr (MM) return half_slope1<true, R>(dl, dr);
    const R a = dl + dr;
    const R m = rmin(rmin(rabs(dl), rabs(dr)), R(0.25) * rabs(a));
    return dl * dr <= R(0) ? R(0) : (a >= R(0) ? m : -m);
}

// predictor: one thread per cell, plane blockIdx.y of the slab's S + 2
template <class R, int RECON> __global__ void __launch_bounds__(128, 3) pass_recon_kernel(const PassArgs<R> P) {
    const UnsplitArgs<R>& A = P.A;
    constexpr bool MM = RECON == RECON_MINMOD;
    const int nx = A.nx, ny = A.ny;
    const size_t nxy = (size_t)nx * ny, qn = nxy * (P.S + 4), mn = nxy * (P.S + 2);
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nxy) return;
    const int k = blockIdx.y;
    const int y = (int)(c / (unsigned)nx), x = (int)(c - (unsigned)y * nx);
    const R* q0 = P.q + (size_t)(k + 1) * nxy;
    const size_t off[6] = {(size_t)y * nx + wrap1(x - 1, nx), (size_t)y * nx + wrap1(x + 1, nx),
                           (size_t)wrap1(y - 1, ny) * nx + x, (size_t)wrap1(y + 1, ny) * nx + x, (size_t)c, (size_t)c};
    const R* row[6] = {q0, q0, q0, q0, q0 - nxy, q0 + nxy};
    Q9<R> m0, s[3];
    bool up = true;
#pragma unroll
    for (int v = 0; v < 9; ++v) m0.v[v] = q0[v * qn + c];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int v = 0; v < 9; ++v) {
            const R l = row[2 * d][v * qn + off[2 * d]], r = row[2 * d + 1][v * qn + off[2 * d + 1]];
            s[d].v[v] = pass_slope<MM>(m0.v[v] - l, r - m0.v[v]);
            if (RECON == RECON_PPM && v == 4) up = up && !spj(l, m0.v[v], r);
        }
    const Consts<R>& K = A.K;
    Q9<R> mh = cons2prim(hancock(m0, s[0], s[1], s[2], step_vals(A).dtdx, K.gamma), K.gamma, K.smallr, K.pfl);
    if (mh.v[0] <= K.smallr || mh.v[4] <= K.pfl) mh = m0;
#pragma unroll
    for (int v = 0; v < 9; ++v) P.mh[v * mn + k * nxy + c] = mh.v[v];
    if (RECON == RECON_PPM) P.up[k * nxy + c] = up;
}

// The two interface states of one face and its flux, in the frame whose x axis is the face normal d:
// component i of that frame is variable rot[i], so the rotation is in the addresses.  c[0..3] are the
// in-slab offsets of the cells -1, 0 | 1, 2 along d, relative to plane zs - 2 (Q); the predictors of
// cells 0 and 1 sit one plane lower in MH.
template <class R, int RECON, int RIEM>
__device__ __forceinline__ Q9<R> pass_face(const PassArgs<R>& P, const StepVals<R>& V, const size_t c[4], size_t nxy,
                                           int d) {
    constexpr bool MM = RECON == RECON_MINMOD;
    const UnsplitArgs<R>& A = P.A;
    const size_t qn = nxy * (P.S + 4), mn = nxy * (P.S + 2);
    const int e1 = d, e2 = d == 2 ? 0 : d + 1, e3 = d == 0 ? 2 : d - 1;
    const int rot[9] = {0, 1 + e1, 1 + e2, 1 + e3, 4, 5 + e1, 5 + e2, 5 + e3, 8};
    bool upl = false, upr = false;
    if (RECON == RECON_PPM) {
        upl = P.up[c[1] - nxy] != 0;
        upr = P.up[c[2] - nxy] != 0;
    }
    Q9<R> L, Rr;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const R* q = P.q + (size_t)rot[i] * qn;
        const R* m = P.mh + (size_t)rot[i] * mn;
        const R a = q[c[0]], b = q[c[1]], e = q[c[2]], f = q[c[3]];
        const R ml = m[c[1] - nxy], mr = m[c[2] - nxy];
        R l = ml + pass_slope<MM>(b - a, e - b), r = mr - pass_slope<MM>(e - b, f - e);
        if (RECON == RECON_PPM) {
            R lo, hi;
            if (upl) {
                ppm_edges(a, b, e, lo, hi);
                l = ml + hi - b;
            }
            if (upr) {
                ppm_edges(b, e, f, lo, hi);
                r = mr + lo - e;
            }
        }
        L.v[i] = l;
        Rr.v[i] = r;
    }
    const Consts<R>& K = A.K;
    if (A.iflo) {   // rare: revert an unphysical state to the cell value
        if (L.v[0] < K.smallr || L.v[4] < K.pfl)
#pragma unroll
            for (int i = 0; i < 9; ++i) L.v[i] = P.q[(size_t)rot[i] * qn + c[1]];
        if (Rr.v[0] < K.smallr || Rr.v[4] < K.pfl)
#pragma unroll
            for (int i = 0; i < 9; ++i) Rr.v[i] = P.q[(size_t)rot[i] * qn + c[2]];
    }
    return riemann_glm<0, RIEM>(L, Rr, K, V.ch, A.use_llf != 0);
}

// Fluxes and update: a block owns TX x TY columns over lz planes and marches z.  Per plane each thread
// solves its cell's upper z, x and y faces, and the first TX + TY threads one face each of the tile's
// low y and low x sides, all by the same code (one copy of the solver for the three directions and the
// boundary: the instruction cache holds it).  Fluxes meet in shared memory; two barriers per plane.
template <int TX, int TY> constexpr size_t pass_flux_smem(size_t real) {
    return 9 * real * ((size_t)(TX + 1) * TY + (size_t)TX * (TY + 1) + 2 * (size_t)TX * TY) + 32 * sizeof(double);
}
template <class R, int RECON, int RIEM, int TX, int TY, int MINB>
__global__ void __launch_bounds__(TX * TY, MINB) pass_flux_kernel(const PassArgs<R> P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NT = TX * TY, NFX = (TX + 1) * TY, NFY = TX * (TY + 1);
    static_assert(NT >= TX + TY && NT % 32 == 0, "one boundary face per thread");
    R* FX = reinterpret_cast<R*>(smem_raw);   // [9][TY][TX + 1]
    R* FY = FX + 9 * NFX;                      // [9][TY + 1][TX]
    R* FZ = FY + 9 * NFY;                      // [2][9][NT]: the z faces below and above, by plane parity
    double* red = reinterpret_cast<double*>(FZ + 18 * NT);
    const UnsplitArgs<R>& A = P.A;
    const StepVals<R> V = step_vals(A);
    const Consts<R>& K = A.K;
    const int nx = A.nx, ny = A.ny;
    const size_t nxy = (size_t)nx * ny;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const int gx = x0 + tx, gy = y0 + ty;
    const bool own = gx < nx && gy < ny;
    const int k0 = blockIdx.z * P.lz, k1 = min(k0 + P.lz, P.S);   // planes of the slab
    // this thread's boundary face: low y side of column tid, low x side of row tid - TX
    const bool by = tid < TX && x0 + tid < nx, bx = tid >= TX && tid < TX + TY && y0 + tid - TX < ny;
    const bool turb = A.do_turb && A.btab != nullptr;
    R cmax = R(0), smax = R(0);
    for (int k = k0 - 1; k < k1; ++k) {
        const int tasks = k < k0 ? 1 : (by || bx ? 4 : 3);
#pragma unroll 1
        for (int t = 0; t < tasks; ++t) {
            // task 0: upper z face, 1: upper x, 2: upper y of the own cell, 3: boundary face
            int d = t == 0 ? 2 : t - 1, x = gx, y = gy;
            R* out;
            int stride;
            if (t < 3) {
                if (!own) continue;
                out = t == 0 ? FZ + 9 * NT * (k & 1) + tid : (t == 1 ? FX + tx + 1 + (TX + 1) * ty : FY + tx + TX * (ty + 1));
                stride = t == 0 ? NT : (t == 1 ? NFX : NFY);
            } else if (by) {
                d = 1; x = x0 + tid; y = y0 == 0 ? ny - 1 : y0 - 1;
                out = FY + tid; stride = NFY;
            } else {
                d = 0; x = x0 == 0 ? nx - 1 : x0 - 1; y = y0 + tid - TX;
                out = FX + (TX + 1) * (tid - TX); stride = NFX;
            }
            // cells -1, 0 | 1, 2 along d in plane k of the slab (plane k + 2 of Q)
            const size_t base = (size_t)(k + 2) * nxy;
            size_t c[4];
            if (d == 2) {
                const size_t g = (size_t)y * nx + x + base;
                c[0] = g - nxy; c[1] = g; c[2] = g + nxy; c[3] = g + 2 * nxy;
            } else if (d == 0) {
                const size_t r = (size_t)y * nx + base;
                const int xp = x + 1 < nx ? x + 1 : 0;
                c[0] = r + (x > 0 ? x - 1 : nx - 1); c[1] = r + x; c[2] = r + xp; c[3] = r + (xp + 1 < nx ? xp + 1 : 0);
            } else {
                const int yp = y + 1 < ny ? y + 1 : 0;
                c[0] = base + x + (size_t)(y > 0 ? y - 1 : ny - 1) * nx; c[1] = base + x + (size_t)y * nx;
                c[2] = base + x + (size_t)yp * nx; c[3] = base + x + (size_t)(yp + 1 < ny ? yp + 1 : 0) * nx;
            }
            const Q9<R> f = pass_face<R, RECON, RIEM>(P, V, c, nxy, d);
            const int e2 = d == 2 ? 0 : d + 1, e3 = d == 0 ? 2 : d - 1;
            out[0] = f.v[0];
            out[(1 + d) * stride] = f.v[1]; out[(1 + e2) * stride] = f.v[2]; out[(1 + e3) * stride] = f.v[3];
            out[4 * stride] = f.v[4];
            out[(5 + d) * stride] = f.v[5]; out[(5 + e2) * stride] = f.v[6]; out[(5 + e3) * stride] = f.v[7];
            out[8 * stride] = f.v[8];
        }
        if (k < k0) continue;
        __syncthreads();
        if (own) {
            const int kz = P.zs + k;
            const size_t g = (size_t)gx + (size_t)nx * gy + nxy * kz;
            const R* fx = FX + tx + (TX + 1) * ty;
            const R* fy = FY + tx + TX * ty;
            const R* fl = FZ + 9 * NT * ((k + 1) & 1) + tid;   // below: written at plane k - 1
            const R* fh = FZ + 9 * NT * (k & 1) + tid;
            Q9<R> q;
#pragma unroll
            for (int v = 0; v < 9; ++v) {
                const R xy = (fx[v * NFX] - fx[v * NFX + 1]) + (fy[v * NFY] - fy[v * NFY + TX]);
                q.v[v] = A.u.p[v][g] + V.dtdx * (xy + (fl[v * NT] - fh[v * NT]));
            }
            R ax = R(0), ay = R(0), az = R(0);
            if (turb) force_accel(A.btab + ((size_t)kz * ny + gy) * 24, A.trigx, nx, gx, V.ramp, ax, ay, az);
            finish_update(q, K, V.glm_fac, turb, ax, ay, az, V.dt);
#pragma unroll
            for (int v = 0; v < 9; ++v) A.o.p[v][g] = q.v[v];
            if (A.cfl_out) {
                R ct, sg;
                cfl_speeds(q, K, ct, sg);
                cmax = rmax(cmax, ct);
                smax = rmax(smax, sg);
            }
        }
        __syncthreads();
    }
    if (A.cfl_out) {
        block_max_atomic((double)cmax, A.cfl_out, red);
        __syncthreads();
        block_max_atomic((double)smax, A.cfl_out + 1, red);
    }
}

}  // namespace gmt
