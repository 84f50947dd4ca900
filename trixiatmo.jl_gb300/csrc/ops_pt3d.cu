#include "ops_3d.cuh"

const Ops* ops_pt3d(int n) { return ops3d_for_n<PhysPT3D>(n); }
