// Face arithmetic of the CloverLeaf advection kernels (2D and the fused
// loops), on values the caller has picked: the operation order is the
// reference's (apps/c/CloverLeaf/advec_cell_kernel.h:28-104,
// advec_mom_kernel.h:139-163).
#pragma once
#include "ops_b200_device.cuh"

namespace opsb {
namespace clover {

// Donor-cell / van Leer mass and energy flux through one face. `pv` is the
// donor's pre-advection volume, `width` the ratio of the face's cell width
// to that of the cell across it, (d, e) the density and energy of the donor,
// upwind and downwind cells.
__device__ __forceinline__ void advec_cell_face(double vol_flux, double pv, double width, double d_don, double d_up,
                                                double d_dwn, double e_don, double e_up, double e_dwn,
                                                double &mass_flux, double &ener_flux) {
  const double one_by_six = 1.0 / 6.0;
  double sigmat = qdiv(fabs(vol_flux), pv);
  double sigma3 = (1.0 + sigmat) * width;
  double sigma4 = 2.0 - sigmat;
  double sigmav = sigmat;
  double diffuw = d_don - d_up;
  double diffdw = d_dwn - d_don;
  double limiter;
  if ((diffuw * diffdw) > 0.0)
    limiter = (1.0 - sigmav) * op_sign(1.0, diffdw) *
              op_min(op_min(fabs(diffuw), fabs(diffdw)), one_by_six * (sigma3 * fabs(diffuw) + sigma4 * fabs(diffdw)));
  else
    limiter = 0.0;
  mass_flux = (vol_flux) * (d_don + limiter);
  double sigmam = qdiv(fabs(mass_flux), d_don * pv);
  diffuw = e_don - e_up;
  diffdw = e_dwn - e_don;
  if ((diffuw * diffdw) > 0.0)
    limiter = (1.0 - sigmam) * op_sign(1.0, diffdw) *
              op_min(op_min(fabs(diffuw), fabs(diffdw)), one_by_six * (sigma3 * fabs(diffuw) + sigma4 * fabs(diffdw)));
  else
    limiter = 0.0;
  ener_flux = mass_flux * (e_don + limiter);
}

// Momentum flux through one node face: `sigma` = |node flux| / donor node
// mass, `width` the cell width at the node, `wdif` that of the cell across,
// v the velocity at the donor, upwind and downwind nodes.
__device__ __forceinline__ double advec_mom_face(double node_flux, double sigma, double width, double wdif,
                                                 double v_don, double v_up, double v_dwn) {
  double vdiffuw = v_don - v_up;
  double vdiffdw = v_dwn - v_don;
  double limiter = 0.0;
  if (vdiffuw * vdiffdw > 0.0) {
    double auw = fabs(vdiffuw);
    double adw = fabs(vdiffdw);
    double wind = 1.0;
    if (vdiffdw <= 0.0) wind = -1.0;
    limiter = wind * op_min(width * ((2.0 - sigma) * adw / width + (1.0 + sigma) * auw / wdif) / 6.0,
                            op_min(auw, adw));
  }
  double advec_vel_temp = v_don + (1.0 - sigma) * limiter;
  return advec_vel_temp * node_flux;
}

}  // namespace clover
}  // namespace opsb
