// fi_engine_wide.cu — the step engine's kernels on register lines, of grids wider than a block.
#define FI_ENGINE_PART 2
#include "fi_engine.cu"
