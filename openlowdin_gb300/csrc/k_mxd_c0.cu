// MP2 transform input in double-float of bra pair class 0 (ss) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_MXD_TABLE(0)
}  // namespace lgb
