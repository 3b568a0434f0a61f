// fi_engine_lines.cu — the step engine's kernels on register lines.
#define FI_ENGINE_PART 1
#include "fi_engine.cu"
