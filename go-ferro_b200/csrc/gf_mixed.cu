// Mixed-precision (FP32) stage sequence of the engine, in a translation unit
// of its own (the two units compile in parallel).  This file instantiates only the <S, float>
// stage kernels and exports gf_mixed_enqueue_step / gf_mixed_elastic_setup,
// declared in gf_engine.cu.
#define GF_MIXED_TU 1
#include "gf_engine.cu"
