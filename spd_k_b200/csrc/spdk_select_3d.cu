// Kernel instantiations of one group of (ndim, p) variants.
#include "spdk_kernelset.cuh"

namespace spdk {

bool select_3d(int p, KernelSetT<double>* k, bool visc) {
    switch (p) {
    case 1: return pick3<double, 1>(k, visc);
    case 2: return pick3<double, 2>(k, visc);
    case 3: return pick3<double, 3>(k, visc);
    case 4: return pick3<double, 4>(k, visc);
    case 5: return pick3<double, 5>(k, visc);
    }
    return false;
}

}  // namespace spdk
