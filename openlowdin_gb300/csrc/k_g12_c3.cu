// geminal (G12) kernels of bra pair class 3 (ds) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_G12_TABLE(3)
}  // namespace lgb
