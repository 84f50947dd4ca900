#include "ops_2d.cuh"

const Ops* ops_ie2d(int n) { return ops_for_n<PhysIE2D>(n); }
