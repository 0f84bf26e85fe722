// Instantiations of the FP32 register-block adjoint.
#include "adj_block.cuh"
#define KGB_D(NN, D) \
    case NN * 16 + D: return adj_info_of<AdjTune<NN, D>>();
namespace kgb {
AdjBlkInfo adj_block_lookup(int n, int d)
{
    if (d < 1 || d > 15) return AdjBlkInfo{};  // the keys below hold d in 4 bits
    switch (n * 16 + d) {
        KGB_D(2, 2) KGB_D(2, 3) KGB_D(2, 4) KGB_D(2, 5) KGB_D(2, 6) KGB_D(2, 7) KGB_D(2, 8)
        KGB_D(3, 2) KGB_D(3, 3) KGB_D(3, 4) KGB_D(3, 5) KGB_D(3, 6)
        KGB_D(4, 2) KGB_D(4, 3) KGB_D(4, 4) KGB_D(4, 5)
        KGB_D(5, 2) KGB_D(5, 3) KGB_D(5, 4) KGB_D(5, 5)
        KGB_D(6, 2) KGB_D(6, 3) KGB_D(6, 4)
        KGB_D(7, 2) KGB_D(7, 3) KGB_D(7, 4)
        KGB_D(8, 2) KGB_D(8, 3) KGB_D(8, 4)
    default: return AdjBlkInfo{};
    }
}
}  // namespace kgb
