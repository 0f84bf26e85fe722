// Instantiations of the deterministic FP64 groups of short vectors (n^d <= 1024).
#include "grouped_f64.cuh"

namespace kgb {

template <int NN, int D> static GqF64Info info()
{
    using K = F64<NN, D>;
    GqF64Info f;
    if constexpr (K::N <= K::threads) f.fn[0] = gq_f64_det_kernel<NN, D, 1>;
    if constexpr (K::N <= 2 * K::threads) f.fn[1] = gq_f64_det_kernel<NN, D, 2>;
    f.fn[2] = gq_f64_det_kernel<NN, D, 4>;
    f.n = NN;
    f.d = D;
    f.threads = K::threads;
    f.entry_bytes = (K::VS + K::FS) * 8 + 8 + 1;  // vector, factors, place, flags
    return f;
}

GqF64Info gq_f64_lookup(int n, int d)
{
    if (d < 1 || d > 15) return GqF64Info{};  // the keys below hold d in 4 bits
    switch (n * 16 + d) {
    case 2 * 16 + 1: return info<2, 1>();
    case 2 * 16 + 2: return info<2, 2>();
    case 2 * 16 + 3: return info<2, 3>();
    case 2 * 16 + 4: return info<2, 4>();
    case 2 * 16 + 5: return info<2, 5>();
    case 2 * 16 + 6: return info<2, 6>();
    case 2 * 16 + 7: return info<2, 7>();
    case 2 * 16 + 8: return info<2, 8>();
    case 2 * 16 + 9: return info<2, 9>();
    case 2 * 16 + 10: return info<2, 10>();
    case 3 * 16 + 1: return info<3, 1>();
    case 3 * 16 + 2: return info<3, 2>();
    case 3 * 16 + 3: return info<3, 3>();
    case 3 * 16 + 4: return info<3, 4>();
    case 3 * 16 + 5: return info<3, 5>();
    case 3 * 16 + 6: return info<3, 6>();
    case 4 * 16 + 1: return info<4, 1>();
    case 4 * 16 + 2: return info<4, 2>();
    case 4 * 16 + 3: return info<4, 3>();
    case 4 * 16 + 4: return info<4, 4>();
    case 4 * 16 + 5: return info<4, 5>();
    case 5 * 16 + 1: return info<5, 1>();
    case 5 * 16 + 2: return info<5, 2>();
    case 5 * 16 + 3: return info<5, 3>();
    case 5 * 16 + 4: return info<5, 4>();
    case 6 * 16 + 1: return info<6, 1>();
    case 6 * 16 + 2: return info<6, 2>();
    case 6 * 16 + 3: return info<6, 3>();
    case 7 * 16 + 1: return info<7, 1>();
    case 7 * 16 + 2: return info<7, 2>();
    case 7 * 16 + 3: return info<7, 3>();
    case 8 * 16 + 1: return info<8, 1>();
    case 8 * 16 + 2: return info<8, 2>();
    case 8 * 16 + 3: return info<8, 3>();
    case 9 * 16 + 1: return info<9, 1>();
    case 9 * 16 + 2: return info<9, 2>();
    case 9 * 16 + 3: return info<9, 3>();
    case 10 * 16 + 1: return info<10, 1>();
    case 10 * 16 + 2: return info<10, 2>();
    case 10 * 16 + 3: return info<10, 3>();
    default: return GqF64Info{};
    }
}

}  // namespace kgb
