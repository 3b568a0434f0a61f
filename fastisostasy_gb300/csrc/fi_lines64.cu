// fi_lines64.cu — the register-line transforms in double precision.
#define FI_LINES_T double
#include "fi_lines.cu"
