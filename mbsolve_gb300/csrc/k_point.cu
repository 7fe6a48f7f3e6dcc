// Cayley kernels of runs of a single grid point in FP64.
#include "inst.cuh"
#include "point_cayley.cuh"

namespace mbg {

template<int LEV>
void launch_point(const kparams<double>& p, unsigned grid, size_t, cudaStream_t s)
{
    point_cayley_kernel<LEV><<<grid, POINT_THREADS, 0, s>>>(p);
}

}  // namespace mbg

#define MBG_REG_POINT(LEV)                                                          \
    static const bool MBG_CAT(mbg_reg_, __LINE__) = ::mbg::register_kernel<double>( \
        ::mbg::ALGO_CAYLEY, LEV, 1, ::mbg::POINT_THREADS, &::mbg::launch_point<LEV>, ::mbg::STAGING_POINT);

MBG_REG_POINT(2)
MBG_REG_POINT(3)
MBG_REG_POINT(4)
MBG_REG_POINT(5)
