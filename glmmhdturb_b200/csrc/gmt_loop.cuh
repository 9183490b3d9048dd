// gmt_loop.cuh -- device-resident time loop: the host loop of run_turb (glmmhd_turb.jl:2216-2230)
// moved onto the GPU so that many steps run without a host round trip and can be captured in a
// CUDA graph.
//
// Per step and per box: the tick kernel turns the CFL maxima that the previous step fused into
// its write-out into dt, ch, glm_fac and the forcing ramp, decides whether the OU forcing advances
// this step (t >= next_time, glmmhd_turb.jl:2217), makes its OU update and clips dt to the forcing
// cadence and t_end (:2221); the conditional mode-table kernel then runs only on boxes that advance,
// and the step kernel reads its dt, ch, glm_fac and ramp from the same record.
#pragma once
#include "gmt_internal.h"

namespace gmt {

// per-box loop record in device memory; dt, ch, glm_fac, ramp first (the step kernel's dparams)
struct LoopState {
    double dt, ch, glm_fac, ramp;
    double t, t_end, next_time;
    uint32_t counter;   // OU updates done
    int advance;        // 1: the forcing advances before this step
    int status;         // 1: no positive finite CFL maximum (state invalid); steps then have dt = 0
    int pad;
};

// per-box constants of the loop
struct LoopConst {
    double courant, dx, boxlen, cp_coef, glm_ch_scale, turb_T, dtf, alpha, beta, sigma0;
    int ch_max_signal;  // 1: ch = global max signal speed; 0: ch = courant*dx/dt/3*glm_ch_scale
    int do_turb;
    uint32_t seed;
    int pad;
};

// One block of 64 threads per box: thread 0 turns the box's CFL maxima into its step values and clears
// them for the step to come; if the forcing advances, the block then makes the OU update of the 61
// modes.  (One launch in the place of a tick, an OU launch and a memset: a 64^3 step takes about 40 us,
// and each of the three cost 2 to 4.)
__global__ void __launch_bounds__(64) tick_kernel(LoopState* st, const LoopConst* cs, unsigned long long* cfl, double* modes,
                                                  const int* mode_k) {
    const int b = blockIdx.x, q = threadIdx.x;
    __shared__ int advance;
    __shared__ uint32_t counter;
    if (q == 0) {
        LoopState S = st[b];
        const LoopConst C = cs[b];
        double cmax = __longlong_as_double((long long)cfl[2 * b]);
        double smax = __longlong_as_double((long long)cfl[2 * b + 1]);
        cfl[2 * b] = cfl[2 * b + 1] = 0ull;
        S.advance = 0;
        if (C.do_turb && S.t >= S.next_time) {
            S.advance = 1;
            S.next_time += C.dtf;
        }
        double dt = 0.0;
        if (cmax > 0.0 && isfinite(cmax)) {
            dt = C.courant * C.dx / cmax;
        } else {
            S.status = 1;
        }
        if (C.do_turb) dt = fmin(dt, S.next_time - S.t);
        dt = fmin(dt, S.t_end - S.t);
        if (!(dt > 0.0)) dt = 0.0;
        double ch = S.ch;
        if (dt > 0.0) ch = C.ch_max_signal ? smax : C.courant * C.dx / dt / 3.0 * C.glm_ch_scale;
        if (!(ch > 0.0)) ch = 1.0;
        S.dt = dt;
        S.ch = ch;
        S.glm_fac = C.cp_coef > 0.0 ? exp(-(ch * ch / (C.cp_coef * C.boxlen * ch)) * dt) : 1.0;
        S.ramp = C.turb_T > 0.0 ? fmin(S.t / C.turb_T, 1.0) : 1.0;
        S.t += dt;
        advance = S.advance;
        counter = S.counter;
        if (S.advance) S.counter = S.counter + 1;
        st[b] = S;
    }
    __syncthreads();
    if (advance && q < 61) {
        const LoopConst& C = cs[b];
        ou_mode_update(modes + (size_t)b * 61 * 6, q, mode_k[3 * q], mode_k[3 * q + 1], mode_k[3 * q + 2], C.seed, counter,
                       C.alpha, C.beta, C.sigma0);
    }
}

// mode-table rows of advancing boxes; grid (rows, boxes)
template <class R> struct BoxTables {
    const double* modes;   // [61][3][2] of this box
    const R* trigy;
    const R* trigz;
    R* btab;
    int ny, nz;
};
template <class R>
__global__ void __launch_bounds__(256) btab_cond_kernel(const BoxTables<R>* bt, const LoopState* st, const int* mode_k) {
    const int b = blockIdx.y;
    if (!st[b].advance) return;
    const BoxTables<R> T = bt[b];
    const int rows = T.ny * T.nz;
    for (int r = (int)blockIdx.x * BTAB_ROWS; r < rows; r += (int)gridDim.x * BTAB_ROWS) {
        btab_rows(T.modes, mode_k, T.trigy, T.trigz, T.ny, T.nz, r, T.btab);
        __syncthreads();   // the shared tables are refilled for the next rows
    }
}

}  // namespace gmt
