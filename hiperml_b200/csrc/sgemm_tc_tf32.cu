// The TF32X3 form's kernels (sgemm_tc.cu), a module of their own.
#define HML_TC_PART 4
#include "sgemm_tc.cu"
