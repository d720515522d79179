// geminal (G12) kernels of bra pair class 2 (pp) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_G12_TABLE(2)
}  // namespace lgb
