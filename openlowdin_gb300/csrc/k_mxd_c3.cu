// MP2 transform input in double-float of bra pair class 3 (ds) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_MXD_TABLE(3)
}  // namespace lgb
