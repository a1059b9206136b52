// FP32 image-formation instantiations: fftsize 8, 10, 12, 16.
#include "wfs_form.cuh"

SHWFS_REGISTER_FORM4(8)
SHWFS_REGISTER_FORM(10)
SHWFS_REGISTER_FORM4(12)
SHWFS_REGISTER_FORM4(16)
