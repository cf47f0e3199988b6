// fz_compress_abs.cu -- the encode kernels of an absolute bound (fz_compress.cuh), compiled beside those
// of a relative one in fz_compress.cu.
#include "fz_compress.cuh"

namespace fz {

EncodeKernel* encode_kernel_abs(int nd, bool list) { return pick_encode_kernel<false>(nd, list); }
WholeKernel*  whole_kernel_abs(int nd, bool scan) { return pick_whole_kernel<false>(nd, scan); }

}  // namespace fz
