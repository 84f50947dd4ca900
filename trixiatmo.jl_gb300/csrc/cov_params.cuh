// Parameters of the covariant shallow-water kernels: the equations' gravity
// and the volume / surface flux choices, and the element groups of a handle
// (see cov_kernels.cuh).
#pragma once

namespace tag {

struct CovParams {
  double g;
  int split;     // SplitCovariantShallowWaterEquations2D
  int volume;    // 0 weak form, 1 flux differencing
  int vol_sym;   // 0 flux_central, 1 flux_ec
  int vol_nc;    // 0 none, 1 flux_nonconservative_ec
  int surf_sym;  // 0 flux_central, 1 flux_ec
  int surf_diss; // 0 none, 1 local Lax-Friedrichs
  int surf_nc;   // 0 none, 1 flux_nonconservative_ec, 2 flux_nonconservative_surface_simplified
};

struct CovGroup {
  int n;         // nodes per direction
  int e0, ne;    // elements [e0, e0 + ne)
  long node0;    // first node of element e0
  long sf0;      // first double of element e0 in the surface-flux array
  int if0, nif;  // interfaces [if0, if0 + nif)
  int epb;       // elements per CTA
  int blk0;      // first CTA of the group in the element launch
  int iblk0;     // first CTA of the group in the interface launch
  long ifnode0;  // first node of interface if0 in the packed interface geometry
  int basis;     // offset of the group's BasisDev in the basis array
};

constexpr int kCovMaxGroups = 64;

struct CovGroups {
  int count;
  CovGroup g[kCovMaxGroups];
};

}  // namespace tag
