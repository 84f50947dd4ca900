#include "ops_2d.cuh"

const Ops* ops_energy2d(int n) { return ops_for_n<PhysEnergy2D>(n); }
