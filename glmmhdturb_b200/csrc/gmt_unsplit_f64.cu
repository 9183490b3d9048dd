// FP64 unsplit step kernels: up to 256 threads, 1 resident block per SM.  Built with --fmad=false
// so each expression rounds exactly as the IEEE evaluation of the oracle.
#include <algorithm>

#include "gmt_passes.cuh"
#include "gmt_unsplit_inst.cuh"

namespace gmt {
// compile-time tiles for the production schemes (constant strides and loop bounds)
template <int TOX, int TOY, bool MAY_OVER>
static bool fixed_tile64(const UnsplitArgs<double>& A, int recon, int riem, cudaStream_t s, cudaError_t& e) {
    if (A.ox != TOX || A.oy != TOY) return false;
#define GMT_FIX(RC, RM) \
    if (recon == RC && riem == RM) { e = unsplit_go<double, RC, RM, 256, 1, TOX, TOY, MAY_OVER>(A, s); return true; }
    GMT_FIX(RECON_MC, RIEM_HLLD) GMT_FIX(RECON_MC, RIEM_HLL) GMT_FIX(RECON_PPM, RIEM_HLL)
#undef GMT_FIX
    return false;
}
cudaError_t launch_unsplit(const UnsplitArgs<double>& A, int recon, int riem, cudaStream_t s) {
    if (A.ox * A.oy > 256) return cudaErrorInvalidConfiguration;
    cudaError_t e = cudaSuccess;
    if (fixed_tile64<32, 8, false>(A, recon, riem, s, e) || fixed_tile64<16, 16, true>(A, recon, riem, s, e)) return e;
    return unsplit_dispatch_t<double, 256, 1>(A, recon, riem, s);
}
cudaError_t launch_batch(const BatchArgs<double>& P, int boxes, int recon, int riem, cudaStream_t s) {
#define GMT_CASE(RC, RM) \
    if (recon == RC && riem == RM) return batch_go<double, RC, RM, 256, 1, 16, 16>(P, boxes, s);
    GMT_CASE(RECON_MC, RIEM_HLLD) GMT_CASE(RECON_MC, RIEM_HLL) GMT_CASE(RECON_PPM, RIEM_HLL)
#undef GMT_CASE
    return cudaErrorNotSupported;
}
// The step as three passes over z slabs of S planes (gmt_passes.cuh); scratch of passes_scratch_bytes.
constexpr int PTX = PASS_TX, PTY = PASS_TY, PMINB = PASS_MINB;
template <int RECON, int RIEM>
static cudaError_t passes_go(const UnsplitArgs<double>& A, void* scratch, int S, cudaStream_t s) {
    const size_t nxy = (size_t)A.nx * A.ny;
    PassArgs<double> P;
    P.A = A;
    const int bx = (A.nx + PTX - 1) / PTX, by = (A.ny + PTY - 1) / PTY;
    for (P.zs = 0; P.zs < A.nz; P.zs += S) {
        P.S = std::min(S, A.nz - P.zs);
        P.q = static_cast<double*>(scratch);
        P.mh = P.q + 9 * nxy * (P.S + 4);
        P.up = reinterpret_cast<unsigned char*>(P.mh + 9 * nxy * (P.S + 2));
        pass_prim_kernel<double><<<dim3((unsigned)((nxy + 255) / 256), P.S + 4), 256, 0, s>>>(P);
        pass_recon_kernel<double, RECON><<<dim3((unsigned)((nxy + 127) / 128), P.S + 2), 128, 0, s>>>(P);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;   // no fluxes from scratch that was not written
        const int lz = P.lz = pass_flux_planes(A.nx, A.ny, P.S);
        pass_flux_kernel<double, RECON, RIEM, PTX, PTY, PMINB>
            <<<dim3(bx, by, (P.S + lz - 1) / lz), PTX * PTY, pass_flux_smem<PTX, PTY>(sizeof(double)), s>>>(P);
    }
    return cudaGetLastError();
}
cudaError_t launch_passes(const UnsplitArgs<double>& A, int recon, int riem, void* scratch, int S, cudaStream_t s) {
#define GMT_CASE(RC, RM) \
    if (recon == RC && riem == RM) return passes_go<RC, RM>(A, scratch, S, s);
    GMT_CASE(RECON_MC, RIEM_HLLD) GMT_CASE(RECON_MC, RIEM_HLL) GMT_CASE(RECON_MC, RIEM_LLF_BOUND)
    GMT_CASE(RECON_MINMOD, RIEM_HLLD) GMT_CASE(RECON_MINMOD, RIEM_HLL) GMT_CASE(RECON_MINMOD, RIEM_LLF_BOUND)
    GMT_CASE(RECON_PPM, RIEM_HLLD) GMT_CASE(RECON_PPM, RIEM_HLL) GMT_CASE(RECON_PPM, RIEM_LLF_BOUND)
#undef GMT_CASE
    return cudaErrorInvalidValue;
}
// registers and dynamic shared memory of the flux pass, the step's longest
int passes_regs(int recon, int riem) {
    cudaFuncAttributes fa{};
    cudaError_t e = cudaErrorInvalidValue;
#define GMT_CASE(RC, RM) \
    if (recon == RC && riem == RM) e = cudaFuncGetAttributes(&fa, pass_flux_kernel<double, RC, RM, PTX, PTY, PMINB>);
    GMT_CASE(RECON_MC, RIEM_HLLD) GMT_CASE(RECON_MC, RIEM_HLL) GMT_CASE(RECON_MC, RIEM_LLF_BOUND)
    GMT_CASE(RECON_MINMOD, RIEM_HLLD) GMT_CASE(RECON_MINMOD, RIEM_HLL) GMT_CASE(RECON_MINMOD, RIEM_LLF_BOUND)
    GMT_CASE(RECON_PPM, RIEM_HLLD) GMT_CASE(RECON_PPM, RIEM_HLL) GMT_CASE(RECON_PPM, RIEM_LLF_BOUND)
#undef GMT_CASE
    return e == cudaSuccess ? fa.numRegs : -1;
}
size_t passes_smem() { return pass_flux_smem<PTX, PTY>(sizeof(double)); }
cudaError_t unsplit_prepare_f64() {
    cudaError_t e = unsplit_configure_all_t<double, 256, 1>();
#define GMT_FIX(RC, RM)                                                                          \
    if (e == cudaSuccess) e = unsplit_configure<double, RC, RM, 256, 1, 32, 8, false>();         \
    if (e == cudaSuccess) e = unsplit_configure<double, RC, RM, 256, 1, 16, 16>();
    GMT_FIX(RECON_MC, RIEM_HLLD) GMT_FIX(RECON_MC, RIEM_HLL) GMT_FIX(RECON_PPM, RIEM_HLL)
#undef GMT_FIX
    UnsplitArgs<double> none{};
    for (int rc = 0; e == cudaSuccess && rc < 2; ++rc) e = march_dispatch_t<double, 256, 1>(none, rc ? RECON_PPM : RECON_MC, 0, true);
    return e;
}
int unsplit_regs_f64(int recon, int riem, int) { return unsplit_regs_of_t<double, 256, 1>(recon, riem); }
cudaError_t launch_march_tiled(const UnsplitArgs<double>& A, int recon, cudaStream_t s) {
    if (A.ox * A.oy > 256) return cudaErrorInvalidConfiguration;
    return march_dispatch_t<double, 256, 1>(A, recon, s, false);
}
int march_tiled_regs(const UnsplitArgs<double>*, int recon, int) { return march_regs_of_t<double, 256, 1>(recon); }
}  // namespace gmt
