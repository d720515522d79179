// geminal (G12) kernels of bra pair class 5 (dd) for every ket pair class.
#include "class_tables.cuh"

namespace lgb {
LGB_G12_TABLE(5)
}  // namespace lgb
