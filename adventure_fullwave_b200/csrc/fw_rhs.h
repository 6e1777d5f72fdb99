// One entry of a point source, for the device.
#pragma once

#include <cstdint>

namespace fw {

struct RhsPoint {
  int64_t dof;     // local DOF (concatenated over the subdomains)
  int64_t to;      // interior row (>= 0), interface slot k as -k - 2, or -1: a Dirichlet DOF
  double re, im;
};

}  // namespace fw
