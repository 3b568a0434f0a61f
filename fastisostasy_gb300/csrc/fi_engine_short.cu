// fi_engine_short.cu — the step engine's kernels on register lines, short ones among them.
#define FI_ENGINE_PART 3
#include "fi_engine.cu"
