// J/K kernels in double-float of bra pair class 2 (pp) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_JKD_TABLE(2)
}  // namespace lgb
