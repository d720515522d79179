// MP2 transform input in double-float of bra pair class 1 (ps) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_MXD_TABLE(1)
}  // namespace lgb
