// Instantiations of the two-pass kernels for FP32 vectors beyond shared memory.
#include "column_kernels.cuh"

namespace kgb {

template <typename TO, int NN> static ColInfo info()
{
    using K = Col<NN>;
    return ColInfo{(const void *)fwd_column_kernel<TO, NN>, K::threads, K::smem, K::cols};
}
template <typename TO> ColInfo col_lookup(int n)
{
    switch (n) {
    case 2: return info<TO, 2>();
    case 3: return info<TO, 3>();
    case 4: return info<TO, 4>();
    case 5: return info<TO, 5>();
    case 6: return info<TO, 6>();
    case 7: return info<TO, 7>();
    case 8: return info<TO, 8>();
    default: return ColInfo{};
    }
}
template ColInfo col_lookup<float>(int n);
template ColInfo col_lookup<double>(int n);

// the fast axes left by pass 2 of the vectors beyond shared memory
BlkInfo units_lookup(int n, int d1)
{
    if (d1 < 1 || d1 > 15) return BlkInfo{};  // the keys below hold d1 in 4 bits
    if (d1 < 1 || d1 > 15) return BlkInfo{};  // the keys below hold d1 in 4 bits
    switch (n * 16 + d1) {
    case 2 * 16 + 8: return blk_info_of<float, BlkLarge<2, 8>, true>();
    case 2 * 16 + 9: return blk_info_of<float, BlkLarge<2, 9>, true>();
    case 2 * 16 + 10: return blk_info_of<float, BlkLarge<2, 10>, true>();
    case 2 * 16 + 11: return blk_info_of<float, BlkLarge<2, 11>, true>();
    case 2 * 16 + 12: return blk_info_of<float, BlkLarge<2, 12>, true>();
    case 3 * 16 + 6: return blk_info_of<float, BlkLarge<3, 6>, true>();
    case 3 * 16 + 7: return blk_info_of<float, BlkLarge<3, 7>, true>();
    case 3 * 16 + 8: return blk_info_of<float, BlkLarge<3, 8>, true>();
    case 4 * 16 + 5: return blk_info_of<float, BlkLarge<4, 5>, true>();
    case 4 * 16 + 6: return blk_info_of<float, BlkLarge<4, 6>, true>();
    case 5 * 16 + 4: return blk_info_of<float, BlkLarge<5, 4>, true>();
    case 5 * 16 + 5: return blk_info_of<float, BlkLarge<5, 5>, true>();
    case 6 * 16 + 4: return blk_info_of<float, BlkLarge<6, 4>, true>();
    case 6 * 16 + 5: return blk_info_of<float, BlkLarge<6, 5>, true>();
    case 7 * 16 + 4: return blk_info_of<float, BlkLarge<7, 4>, true>();
    case 8 * 16 + 3: return blk_info_of<float, BlkLarge<8, 3>, true>();
    case 8 * 16 + 4: return blk_info_of<float, BlkLarge<8, 4>, true>();
    default: return BlkInfo{};
    }
}

}  // namespace kgb
