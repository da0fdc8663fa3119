// Curvilinear (topography) velocity and stress kernels of the top grid.
#pragma once

#include <cuda_runtime.h>

#include "awp_common.h"
#include "awp_tma.cuh"

struct TopoArgs {
  // wavefield and memory variables (padded layout of awp_common.h)
  float *u1, *v1, *w1, *xx, *yy, *zz, *xy, *xz, *yz;
  float *r1, *r2, *r3, *r4, *r5, *r6;
  // media (rho, 1/lambda, 1/mu, 1/Qp, 1/Qs) and the sponge
  const float *d1, *lam, *mu, *qp, *qs, *dcrjx, *dcrjy, *dcrjz;
  // metrics: 2-D f arrays (ld = ny + 4 + 2 ngsl + 2 align) and 1-D g arrays
  const float *f, *f_1, *f_2, *f_c, *f1_1, *f1_2, *f1_c, *f2_1, *f2_2, *f2_c;
  const float *g, *g_c, *g3, *g3_c;
  AwpTexture tex;
  AwpRelaxTab rel;  // per texture entry, with this struct's DT and 1/h
  int nx, ny, nz, slice, yline, fld;
  float nu;              // velocity: dt/h (topo_t.dth)
  float DT, dth, dh1;    // stress: (dt/h)*h, DT/h, 1/h (topo_set_constants)
  unsigned thr;          // Q(f) switch on a pair sum of Q^-1 (StrArgs::thr)
  int s_i, e_i, s_j, e_j;  // stress window, relative indices, ends exclusive
  // > 0 on a block over a coarser one: level 2, the interface layer, is updated
  // to second order too (dvelc2; dstrqc2 inside the stress window, with the
  // run's own DT, DT/h and 1/h)
  int layer;
  AwpRelaxTab lay_rel;
  AwpLayerTab lay;
  float lay_dt, lay_dth;
};

// dtopo_vel_111_unroll + dtopo_vel_112 (velocity_unroll.cu, optimized_velocity.cu:1040-1629)
// tensor maps: the TmaMaps groups of the velocity and stress kernels with the
// boxes of awp_topo_box (kernel 0: velocity, 1: stress; group 0: j halo, 1:
// media, 2: own); ichunk: x planes a CTA marches at most
int awp_topo_box(int kernel, int group, int* box_x, int* box_y);
cudaError_t awp_launch_topo_velocity(const TopoArgs& a, const TmaMaps& tm, int ichunk, int* err,
                                     cudaStream_t st);
// dtopo_str_111 + dtopo_str_112 (kernels/stress_attenuation.cu:73-1415)
cudaError_t awp_launch_topo_stress(const TopoArgs& a, const TmaMaps& tm, bool elastic, int ichunk,
                                   int* err, cudaStream_t st);
