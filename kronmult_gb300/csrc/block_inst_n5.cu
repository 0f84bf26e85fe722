// Instantiations of the FP32 register-block forward for n = 5.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 5,
          KGB_BLK_D(float, 5, 1)
          KGB_BLK_D(float, 5, 2)
          KGB_BLK_D(float, 5, 3)
          KGB_BLK_D(float, 5, 4)
          KGB_BLK_D(float, 5, 5))
KGB_BLK_N(double, 5,
          KGB_BLK_D(double, 5, 2)
          KGB_BLK_D(double, 5, 3)
          KGB_BLK_D(double, 5, 4)
          KGB_BLK_D(double, 5, 5))
}  // namespace kgb
