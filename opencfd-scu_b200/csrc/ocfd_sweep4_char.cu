// ocfd_sweep4_char.cu -- the in-line walk's instances for WENO7-SYMBO, on the
// characteristic fields and on the flux components.
#include "ocfd_sweep4.cuh"

namespace ocfd {

cudaError_t sweep4_dir_symbo(const Params &p, int dir, cudaStream_t st) {
    return p.charteric ? walk4::dir4_more<walk4::K_SYMC>(p, dir, st) : walk4::dir4_more<walk4::K_SYM>(p, dir, st);
}

}  // namespace ocfd
