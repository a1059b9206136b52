// FP32 image-formation instantiations: fftsize 50, 60, 64.
#include "wfs_form.cuh"

SHWFS_REGISTER_FORM(50)
SHWFS_REGISTER_FORM4(60)
SHWFS_REGISTER_FORM4(64)
