// geminal (G12) kernels of bra pair class 4 (dp) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_G12_TABLE(4)
}  // namespace lgb
