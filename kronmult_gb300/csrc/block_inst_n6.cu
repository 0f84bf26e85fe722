// Instantiations of the FP32 register-block forward for n = 6.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 6,
          KGB_BLK_D(float, 6, 1)
          KGB_BLK_D(float, 6, 3)
          KGB_BLK_D(float, 6, 4)
          KGB_BLK_D(float, 6, 5))
KGB_BLK_N(double, 6,
          KGB_BLK_D(double, 6, 3)
          KGB_BLK_D(double, 6, 4)
          KGB_BLK_D(double, 6, 5))
}  // namespace kgb
