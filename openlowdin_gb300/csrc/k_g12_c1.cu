// geminal (G12) kernels of bra pair class 1 (ps) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_G12_TABLE(1)
}  // namespace lgb
