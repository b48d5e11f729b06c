// Kernel arguments of the diffusion tensor and the tile of one bead pair,
// shared by the stored-tensor build (tensor.cu) and the matrix-free pair
// sums (tea.cu).
#pragma once

#include "bdb_common.cuh"
#include "rpy_tile.cuh"

namespace bdb {

struct TensorArgs {
    int n, npad;
    double preDii, preDij;
    int ewald;
    EwaldConst ec;
};

int ewald_tables(bdb_system* s);          // lattice tables of the Ewald sums (tensor.cu)
TensorArgs targs(const bdb_system* s);

template <typename T, bool kEwald>
__device__ __forceinline__ void tile_of_k(const TensorArgs& A, const double4* pos, int i, int j, T* t)
{
    const double4 pi = pos[i], pj = pos[j];
    if constexpr (kEwald) {
        double d[6];
        rpy_ewald<sizeof(T) == 4>(pi, pj, i == j, A.preDii, A.preDij, A.ec, d);
        for (int k = 0; k < 6; ++k) t[k] = (T)d[k];
    } else if (i == j) {
        const T d = (T)(A.preDii / pi.w);
        t[0] = t[1] = t[2] = d;
        t[3] = t[4] = t[5] = 0;
    } else if (i > j) {
        rpy_free<T>(pi, pj, (T)A.preDii, (T)A.preDij, t);
    } else {
        rpy_free<T>(pj, pi, (T)A.preDii, (T)A.preDij, t);
    }
}

template <typename T>
__device__ __forceinline__ void tile_of(const TensorArgs& A, const double4* pos, int i, int j, T* t)
{
    if (A.ewald)
        tile_of_k<T, true>(A, pos, i, j, t);
    else
        tile_of_k<T, false>(A, pos, i, j, t);
}

}  // namespace bdb
