// Instantiations of the FP32 register-block forward for n = 9.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 9,
          KGB_BLK_D(float, 9, 1)
          KGB_BLK_D(float, 9, 2)
          KGB_BLK_D(float, 9, 3)
          KGB_BLK_D(float, 9, 4))
KGB_BLK_N(double, 9,
          KGB_BLK_D(double, 9, 1)
          KGB_BLK_D(double, 9, 2)
          KGB_BLK_D(double, 9, 3)
          KGB_BLK_D(double, 9, 4))
}  // namespace kgb
