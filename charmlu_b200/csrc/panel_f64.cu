// The FP64 instances of the panel leaf.
#include "panel.cuh"

namespace lub {
LUB_INSTANTIATE_LEAF(double)
}  // namespace lub
