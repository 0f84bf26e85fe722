// Instantiations of the FP32 register-block forward for n = 3.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 3,
          KGB_BLK_D(float, 3, 1)
          KGB_BLK_D(float, 3, 2)
          KGB_BLK_D(float, 3, 3)
          KGB_BLK_D(float, 3, 4)
          KGB_BLK_D(float, 3, 5)
          KGB_BLK_D(float, 3, 6)
          KGB_BLK_D(float, 3, 7)
          KGB_BLK_D(float, 3, 8))
KGB_BLK_N(double, 3,
          KGB_BLK_D(double, 3, 2)
          KGB_BLK_D(double, 3, 4)
          KGB_BLK_D(double, 3, 5)
          KGB_BLK_D(double, 3, 6)
          KGB_BLK_D(double, 3, 7)
          KGB_BLK_D(double, 3, 8))
}  // namespace kgb
