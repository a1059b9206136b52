// FP32 image-formation instantiations: fftsize 32, 40, 48.
#include "wfs_form.cuh"

SHWFS_REGISTER_FORM4(32)
SHWFS_REGISTER_FORM4(40)
SHWFS_REGISTER_FORM4(48)
