#include "ops_3d.cuh"

const Ops* ops_energy3d(int n) { return ops3d_for_n<PhysEnergy3D>(n); }
