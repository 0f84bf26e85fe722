// Instantiations of the FP32 register-block forward for n = 8.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 8,
          KGB_BLK_D(float, 8, 1)
          KGB_BLK_D(float, 8, 2)
          KGB_BLK_D(float, 8, 3)
          KGB_BLK_D(float, 8, 4))
KGB_BLK_N(double, 8,
          KGB_BLK_D(double, 8, 1)
          KGB_BLK_D(double, 8, 2)
          KGB_BLK_D(double, 8, 3)
          KGB_BLK_D(double, 8, 4))
}  // namespace kgb
