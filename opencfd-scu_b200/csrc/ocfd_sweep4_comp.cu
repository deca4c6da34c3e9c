// ocfd_sweep4_comp.cu -- the in-line walk's instances for the schemes on the
// flux components other than WENO7: WENO5, NND2, OMP6, the hybrid scheme
// without projection.
#include "ocfd_sweep4.cuh"

namespace ocfd {

cudaError_t sweep4_dir_comp(const Params &p, int dir, cudaStream_t st) {
    switch (p.scheme_invis) {
    case 302: return walk4::dir4_more<walk4::K_W5>(p, dir, st);
    case 306: return walk4::dir4_more<walk4::K_NND2>(p, dir, st);
    case 310: return walk4::dir4_more<walk4::K_HYBN>(p, dir, st);
    default: return walk4::dir4_more<walk4::K_OMP6>(p, dir, st);
    }
}

}  // namespace ocfd
