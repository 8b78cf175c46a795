// pt_engine_multi.cu -- the engine's variants for blocks that hold several
// replicas, compiled beside the others.
#define PTICM_ENGINE_MULTI
#include "pt_engine.cu"
