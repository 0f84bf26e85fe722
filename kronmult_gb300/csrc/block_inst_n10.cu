// Instantiations of the FP32 register-block forward for n = 10.
#include "block_kernels.cuh"
namespace kgb {
KGB_BLK_N(float, 10,
          KGB_BLK_D(float, 10, 1)
          KGB_BLK_D(float, 10, 2)
          KGB_BLK_D(float, 10, 3)
          KGB_BLK_D(float, 10, 4))
KGB_BLK_N(double, 10,
          KGB_BLK_D(double, 10, 1)
          KGB_BLK_D(double, 10, 2)
          KGB_BLK_D(double, 10, 3)
          KGB_BLK_D(double, 10, 4))
}  // namespace kgb
