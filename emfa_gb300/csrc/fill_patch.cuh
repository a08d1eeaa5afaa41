// Fill by patches of RWGs (fill_patch.cu): the FP64 fills and the
// configuration's 7 x 7-point fill.
#pragma once
#include "emfa_internal.cuh"
#include "fill_entry.cuh"

namespace emfa {

// Fills Z from the self-term table `tab` (the singular table, or the
// configuration's with the triangles' neighbours in g->nbr).  *done false: the
// geometry or the parameters are not for this fill, or there is no room for its
// plan (24 bytes an RWG); nothing was launched.
template <typename T>
emfa_status_t launch_fill_patch(Ctx* c, Geom* g, const GeomDev<T>& d, const emfa_fill_params_t* p,
                                const FillConst<T>& fc, const double2* tab, void* Z, size_t ldz, cudaStream_t st,
                                bool* done);

// slot of triangle ts in the configuration's table of triangle tf: 0 itself,
// 1..3 its edge neighbours, -1 a regular pair
__device__ __forceinline__ int table_slot(const int* __restrict__ nbr, int tf, int ts)
{
    return ts == tf ? 0
           : nbr[3 * (size_t)tf] == ts ? 1
           : nbr[3 * (size_t)tf + 1] == ts ? 2
           : nbr[3 * (size_t)tf + 2] == ts ? 3 : -1;
}

}  // namespace emfa
