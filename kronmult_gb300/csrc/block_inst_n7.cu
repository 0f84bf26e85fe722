// Instantiations of the FP32 register-block forward for n = 7.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 7,
          KGB_BLK_D(float, 7, 1)
          KGB_BLK_D(float, 7, 2)
          KGB_BLK_D(float, 7, 3)
          KGB_BLK_D(float, 7, 4)
          KGB_BLK_D(float, 7, 5))
KGB_BLK_N(double, 7,
          KGB_BLK_D(double, 7, 2)
          KGB_BLK_D(double, 7, 3)
          KGB_BLK_D(double, 7, 4)
          KGB_BLK_D(double, 7, 5))
}  // namespace kgb
