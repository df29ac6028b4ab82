// bl_kernels.cu -- the translation unit holding every hot-path kernel.
// Compiled three times, with -DBL_NS=fast and =mixed (--fmad=true) and
// -DBL_NS=exact (--fmad=false); see bl_kernels.h.
#ifndef BL_NS
#error "compile with -DBL_NS=fast, -DBL_NS=mixed or -DBL_NS=exact"
#endif
#include "hydro_kernels.cuh"
#include "ale_kernels.cuh"
