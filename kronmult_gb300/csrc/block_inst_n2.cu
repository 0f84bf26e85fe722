// Instantiations of the FP32 register-block forward for n = 2 (FP32 outputs).
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 2,
          KGB_BLK_D(float, 2, 1)
          KGB_BLK_D(float, 2, 2)
          KGB_BLK_D(float, 2, 3)
          KGB_BLK_D(float, 2, 4)
          KGB_BLK_D(float, 2, 5)
          KGB_BLK_D(float, 2, 6)
          KGB_BLK_D(float, 2, 7)
          KGB_BLK_D(float, 2, 8)
          KGB_BLK_D(float, 2, 9)
          KGB_BLK_D(float, 2, 10)
          KGB_BLK_D(float, 2, 11)
          KGB_BLK_D(float, 2, 12))
}  // namespace kgb
