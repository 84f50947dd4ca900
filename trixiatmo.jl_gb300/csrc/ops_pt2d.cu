#include "ops_2d.cuh"

const Ops* ops_pt2d(int n) { return ops_for_n<PhysPT2D>(n); }
