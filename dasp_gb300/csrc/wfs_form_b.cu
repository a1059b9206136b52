// FP32 image-formation instantiations: fftsize 20, 24, 30.
#include "wfs_form.cuh"

SHWFS_REGISTER_FORM4(20)
SHWFS_REGISTER_FORM4(24)
SHWFS_REGISTER_FORM(30)
