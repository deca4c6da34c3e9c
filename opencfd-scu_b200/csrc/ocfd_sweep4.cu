// ocfd_sweep4.cu -- the in-line walk's entry points and its FP64 instances
// (the kernels are in ocfd_sweep4.cuh; FP32 instances in ocfd_sweep4_f32.cu).
#include "ocfd_sweep4.cuh"

namespace ocfd {

cudaError_t sweep4_dir_f32(const Params &p, int dir, cudaStream_t st);
cudaError_t sweep4_dir_symbo(const Params &p, int dir, cudaStream_t st);
cudaError_t sweep4_dir_comp(const Params &p, int dir, cudaStream_t st);

// the schemes of sweep variant 6 and of the precision form: the hybrid scheme
// with characteristic projection, WENO7 on the flux components
bool sweeps4_supported(const Params &p) {
    return (p.scheme_invis == 310 && p.charteric) || (p.scheme_invis == 303 && !p.charteric);
}

// Every scheme that walks in line by default: those and, in FP64, all others
// but UP7 and the hybrid scheme by components with one flag for all (mostly
// UP7 faces: the UP7 walk) and the schemes that the reference gives no
// fluxes with projection on.  The generic walk forms a face out of
// line, its loop state in local memory around the call: OMP6 box 97x65x51, two
// steps, 2.24 -> 1.42 ms; characteristic SYMBO box 121x83x47, one, 4.71 -> 1.88.
bool sweeps4_covers(const Params &p) {
    if (sweeps4_supported(p)) return true;
    const int s = p.scheme_invis;
    if (p.mixed || s < 302 || s > 310) return false;
    if (s == 310) return !p.charteric && p.nochar_comp_flag;
    return !p.charteric || s == 304 || s == 305;
}

// one direction of the walk (one kernel); FP32 in the precision form
cudaError_t launch_sweep4_dir(const Params &p, int dir, cudaStream_t st) {
    if (!sweeps4_covers(p)) return cudaErrorNotSupported;
    if (!sweeps4_supported(p))
        return p.scheme_invis == 304 || p.scheme_invis == 305 ? sweep4_dir_symbo(p, dir, st) : sweep4_dir_comp(p, dir, st);
    return p.mixed ? sweep4_dir_f32(p, dir, st) : walk4::dir4r<double>(p, dir, st);
}

cudaError_t launch_sweeps4(const Params &p, cudaStream_t st) {
    if (!sweeps4_supported(p)) return cudaErrorNotSupported;
    cudaError_t e;
    for (int d = 0; d < 3; d++)
        if ((e = launch_sweep4_dir(p, d, st)) != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace ocfd
