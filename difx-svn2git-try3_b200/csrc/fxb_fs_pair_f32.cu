// F stage of two-band work items, FP32 spectra (see fxb_fstage_pair.cuh).
#include "fxb_fstage_pair.cuh"

namespace fxb {

void launch_fs_pair_f32(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	if(k.muxraw)
		launch_var<false, 1>(k, a, stream);
	else if(k.cplx)
		launch_var<false, 2>(k, a, stream);
	else
		launch_var<false, 0>(k, a, stream);
}

}  // namespace fxb
