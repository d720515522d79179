// MP2 transform input in double-float of bra pair class 2 (pp) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_MXD_TABLE(2)
}  // namespace lgb
