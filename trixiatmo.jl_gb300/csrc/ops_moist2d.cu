#include "ops_2d.cuh"

const Ops* ops_moist2d(int n, bool weak) {
  return weak ? ops_for_n<PhysMoist2D, kVolWeak>(n) : ops_for_n<PhysMoist2D, kVolFluxDiff>(n);
}
