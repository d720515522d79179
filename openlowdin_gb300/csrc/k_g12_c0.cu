// geminal (G12) kernels of bra pair class 0 (ss) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_G12_TABLE(0)
}  // namespace lgb
