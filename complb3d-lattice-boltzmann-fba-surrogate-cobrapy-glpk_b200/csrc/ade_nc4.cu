// ade_nc4.cu -- instantiations of the fused transport step with 4 equilibrium
// components (0: no equilibrium), one translation unit per count so they build in parallel.
#include "ade_kernels.cuh"
#include "ops.cuh"

namespace cl {

int ade_step_nc4(Ctx* c) {
    switch (c->ap.n_mob) {
        case 1: return launch_step<1, 4>(c);
        case 2: return launch_step<2, 4>(c);
        case 3: return launch_step<3, 4>(c);
        case 4: return launch_step<4, 4>(c);
        case 5: return launch_step<5, 4>(c);
        case 6: return launch_step<6, 4>(c);
        case 7: return launch_step<7, 4>(c);
        case 8: return launch_step<8, 4>(c);
        default: set_error("the fused transport step supports 1..8 mobile solutes");
                 return CL_ERR_ARG;
    }
}

int ade_ops_nc4(Ctx* c, const AdeK& k, int ops) { return launch_ops<4>(c, k, ops); }

}  // namespace cl
