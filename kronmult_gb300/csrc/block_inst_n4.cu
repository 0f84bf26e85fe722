// Instantiations of the FP32 register-block forward for n = 4.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 4,
          KGB_BLK_D(float, 4, 1)
          KGB_BLK_D(float, 4, 2)
          KGB_BLK_D(float, 4, 3)
          KGB_BLK_D(float, 4, 4)
          KGB_BLK_D(float, 4, 5)
          KGB_BLK_D(float, 4, 6)
          KGB_BLK_D(float, 4, 7))
KGB_BLK_N(double, 4,
          KGB_BLK_D(double, 4, 2)
          KGB_BLK_D(double, 4, 3)
          KGB_BLK_D(double, 4, 4)
          KGB_BLK_D(double, 4, 5)
          KGB_BLK_D(double, 4, 7))
}  // namespace kgb
