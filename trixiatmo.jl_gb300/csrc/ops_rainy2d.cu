#include "ops_2d.cuh"

const Ops* ops_rainy2d(int n, bool weak) {
  return weak ? ops_for_n<PhysRainy2D, kVolWeak>(n) : ops_for_n<PhysRainy2D, kVolFluxDiff>(n);
}
