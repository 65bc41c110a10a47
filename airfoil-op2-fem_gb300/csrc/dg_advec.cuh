// Scalar advection app (advec/src/advec.cpp:171-262) on the device.  Included at the end of
// dg_solver.cu: it shares the per-order operators [Drw | Dsw | -LIFT/2] in constant memory, the
// reference-node coordinates, the affine geometry kernel and the edge records of the Euler path.
//
// One classical RK4 stage is one kernel, advec_fused_kernel (below).  The forms that element-kernel
// forms 0 and (at N = 3) 1 select have two:
//   advec_face_kernel  one thread per face node (boundary faces first): the Lax-Friedrichs flux
//                      n.(F- + F+)/2 + |v|(q- - q+)/2 of advec/src/advec_rhs.h:36-63 once per
//                      face node, with the trace of the neighbour (advec/src/get_neighbour_q.h)
//                      or the constant ghost value 4.5e-5 (advec/src/get_bedge_q.h), written
//                      into both cells' face slots scaled by each side's fscale (twice the flux:
//                      the 1/2 is in the operator's LIFT columns);
//   advec_elem_kernel  32 cells x Np node-warps (even/odd form advec_elem_kernel_sym):
//                      rhs = cr Drw q + cs Dsw q - LIFT flux with
//                      cr = vx rx + vy ry, cs = vx sx + vy sy (F = vx q, G = vy q on affine
//                      cells; advec_rhs.h:11-34), then the RK4 combine: W = q + dt frac k for
//                      stages 0-2 (advec/src/set_workingQ.h) with frac {1/2, 1/2, 1}, and
//                      q += dt/6 (k1 + 2 k2 + 2 k3 + k4) in the last (advec/src/update_Q.h).
//                      k1 + 2 k2 + 2 k3 is accumulated in one array in the reference's order.
// Layout: q, W, acc [K][Np]; flux [K][3][Nfp].  dt is fixed; t is kept on the host.
#pragma once

#include <type_traits>

#include "dg_advec.h"

namespace dg {

constexpr double kAdvecGhost = 4.5e-5;  // advec/src/get_bedge_q.h:10

template <int N>
__global__ void __launch_bounds__(256) advec_face_kernel(const AdvInst d) {
  constexpr int Np = np_of(N), Nfp = N + 1;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nbf = d.nB * Nfp;
  if (tid >= nbf + d.nE * Nfp) return;
  const double vx = d.vx, vy = d.vy, a = d.speed;
  if (tid >= nbf) {
    const int e = (tid - nbf) / Nfp, i = (tid - nbf) - e * Nfp;
    const int4 ed = __ldg(&d.edges[e]);
    const int cL = ed.x, cR = ed.y, fL = ed.z & 3, fR = (ed.z >> 2) & 3;
    const int iR = (ed.z >> 4) ? Nfp - 1 - i : i;
    const double qm = d.W[(size_t)cL * Np + __ldg(&d.fmask[fL * Nfp + i])];
    const double qp = d.W[(size_t)cR * Np + __ldg(&d.fmask[fR * Nfp + iR])];
    const double *gl = d.geo + (size_t)cL * 16 + 4 + 3 * fL;
    const double nx = __ldg(gl), ny = __ldg(gl + 1);
    const double f = nx * (vx * qm + vx * qp) + ny * (vy * qm + vy * qp) + a * (qm - qp);
    d.flux[((size_t)cL * 3 + fL) * Nfp + i] = __ldg(gl + 2) * f;
    d.flux[((size_t)cR * 3 + fR) * Nfp + iR] = -__ldg(d.geo + (size_t)cR * 16 + 6 + 3 * fR) * f;
  } else {
    const int b = tid / Nfp, i = tid - b * Nfp;
    const int4 bd = __ldg(&d.bedges[b]);
    const int c = bd.x, fc = bd.y;
    const double qm = d.W[(size_t)c * Np + __ldg(&d.fmask[fc * Nfp + i])], qp = kAdvecGhost;
    const double *g = d.geo + (size_t)c * 16 + 4 + 3 * fc;
    const double nx = __ldg(g), ny = __ldg(g + 1);
    const double f = nx * (vx * qm + vx * qp) + ny * (vy * qm + vy * qp) + a * (qm - qp);
    d.flux[((size_t)c * 3 + fc) * Nfp + i] = __ldg(g + 2) * f;
  }
}

// stage 0..3: RK4 stage; stage 4: rhs_out = L(W) only.
template <int N>
__global__ void __launch_bounds__(32 * np_of(N)) advec_elem_kernel(const AdvInst d, const int stage) {
  constexpr int Np = np_of(N), NF = 3 * (N + 1), NK = nk_of(N), LD = 33;
  __shared__ double X[(Np + NF) * LD];  // [k][cell]: the tile's W, then its face fluxes
  __shared__ double R[32 * Np];         // right-hand sides, [cell][node] as in HBM
  const int t = threadIdx.x;
  const int e0 = blockIdx.x * 32;
  const int nc = min(32, d.K - e0);
  const size_t base = (size_t)e0 * Np;
  // coalesced loads of the tile's contiguous W and flux ranges
  {
    const int el = t / Np, k = t - el * Np;
    X[k * LD + el] = el < nc ? d.W[base + t] : 0.0;
    for (int j = t; j < 32 * NF; j += 32 * Np) {
      const int ef = j / NF, f = j - ef * NF;
      X[(Np + f) * LD + ef] = ef < nc ? d.flux[(size_t)e0 * NF + j] : 0.0;
    }
  }
  __syncthreads();
  {
    const int lane = t & 31, i = t >> 5;
    double ar = 0.0, as = 0.0, al = 0.0;
#pragma unroll
    for (int k = 0; k < Np; k++) {
      const double x = X[k * LD + lane];
      ar = fma(opA<N>(i * NK + k), x, ar);
      as = fma(opA<N>(i * NK + Np + k), x, as);
    }
#pragma unroll
    for (int f = 0; f < NF; f++) al = fma(opA<N>(i * NK + 2 * Np + f), X[(Np + f) * LD + lane], al);
    double cr = 0.0, cs = 0.0;
    if (lane < nc) {
      const double *g = d.geo + (size_t)(e0 + lane) * 16;
      cr = d.vx * g[0] + d.vy * g[1];
      cs = d.vx * g[2] + d.vy * g[3];
    }
    R[lane * Np + i] = fma(cr, ar, fma(cs, as, al));
  }
  __syncthreads();
  const int el = t / Np;
  if (el >= nc) return;
  const size_t o = base + t;
  const double r = R[t];
  if (stage == 4) {
    d.rhs_out[o] = r;
    return;
  }
  const double q = d.q[o], dt = d.dt;
  // the reference's operation order: q + (dt * frac) * k and q + ((1/6) dt) (((k1 + 2 k2) + 2 k3) + k4)
  if (stage == 0) {
    d.acc[o] = r;
    d.W[o] = __dadd_rn(q, __dmul_rn(dt * 0.5, r));
  } else if (stage < 3) {
    d.acc[o] = __dadd_rn(d.acc[o], 2.0 * r);
    d.W[o] = __dadd_rn(q, __dmul_rn(stage == 1 ? dt * 0.5 : dt, r));
  } else {
    const double qn = __dadd_rn(q, __dmul_rn((1.0 / 6.0) * dt, __dadd_rn(d.acc[o], r)));
    d.q[o] = qn;
    d.W[o] = qn;
  }
}

// The element kernel in even/odd form (the reflection r <-> s splits [Drw | Dsw | -LIFT] into an
// even and an odd block; see elem_tile_sym in dg_solver.cu): the inputs [cr q; cs q; flux] are
// staged in the pair order of that split, added and subtracted pairwise, contracted with the
// even and odd blocks (about half the multiply-adds of the dense rows) and recombined.  Same
// right-hand side as advec_elem_kernel up to rounding; the RK4 combine is the same.
template <int N>
__global__ void __launch_bounds__(32 * np_of(N)) advec_elem_kernel_sym(const AdvInst d, const int stage) {
  constexpr int Np = np_of(N), NF = 3 * (N + 1), NK = nk_of(N), LD = 33;
  constexpr int NUe = Sym<N>::NUe, NUo = Sym<N>::NUo, NRe = Sym<N>::NRe;
  __shared__ double X[NK * LD];   // [slot][cell]
  __shared__ double Y[Np * LD];   // even / odd row results [row][cell]
  __shared__ double R[32 * Np];   // right-hand sides [cell][node]
  const int t = threadIdx.x;
  const int e0 = blockIdx.x * 32;
  const int nc = min(32, d.K - e0);
  const size_t base = (size_t)e0 * Np;
  {
    const int el = t / Np, k = t - el * Np;
    double cr = 0.0, cs = 0.0, w = 0.0;
    if (el < nc) {
      const double *g = d.geo + (size_t)(e0 + el) * 16;
      cr = d.vx * g[0] + d.vy * g[1];
      cs = d.vx * g[2] + d.vy * g[3];
      w = d.W[base + t];
    }
    X[c_pos[N][k] * LD + el] = cr * w;
    X[c_pos[N][Np + k] * LD + el] = cs * w;
    for (int j = t; j < 32 * NF; j += 32 * Np) {
      const int ef = j / NF, f = j - ef * NF;
      X[c_pos[N][2 * Np + f] * LD + ef] = ef < nc ? d.flux[(size_t)e0 * NF + j] : 0.0;
    }
  }
  __syncthreads();
  for (int j = t; j < NUo * 32; j += 32 * Np) {  // butterfly over the input pairs
    const int p = j >> 5, el = j & 31;
    const double a = X[p * LD + el], b = X[(NUe + p) * LD + el];
    X[p * LD + el] = a + b;
    X[(NUe + p) * LD + el] = a - b;
  }
  __syncthreads();
  const int lane = t & 31, i = t >> 5;
  {
    double acc = 0.0;
    if (i < NRe) {
#pragma unroll
      for (int k = 0; k < NUe; k++) acc = fma(opS<N>(i * NUe + k), X[k * LD + lane], acc);
    } else {
#pragma unroll
      for (int k = 0; k < NUo; k++) acc = fma(opS<N>(NRe * NUe + (i - NRe) * NUo + k), X[(NUe + k) * LD + lane], acc);
    }
    Y[i * LD + lane] = acc;
  }
  __syncthreads();
  {
    const int re = c_out[N][3 * i], ro = c_out[N][3 * i + 1], sg = c_out[N][3 * i + 2];
    double r = Y[re * LD + lane];
    if (ro >= 0) r = sg > 0 ? r + Y[ro * LD + lane] : r - Y[ro * LD + lane];
    R[lane * Np + i] = r;
  }
  __syncthreads();
  const int el = t / Np;
  if (el >= nc) return;
  const size_t o = base + t;
  const double r = R[t];
  if (stage == 4) {
    d.rhs_out[o] = r;
    return;
  }
  const double q = d.q[o], dt = d.dt;
  if (stage == 0) {
    d.acc[o] = r;
    d.W[o] = __dadd_rn(q, __dmul_rn(dt * 0.5, r));
  } else if (stage < 3) {
    d.acc[o] = __dadd_rn(d.acc[o], 2.0 * r);
    d.W[o] = __dadd_rn(q, __dmul_rn(stage == 1 ? dt * 0.5 : dt, r));
  } else {
    const double qn = __dadd_rn(q, __dmul_rn((1.0 / 6.0) * dt, __dadd_rn(d.acc[o], r)));
    d.q[o] = qn;
    d.W[o] = qn;
  }
}

// One RK4 stage in one kernel, the contraction on the tensor cores (the exact integer product of
// dg_ozaki.cuh; dense rows at N = 1, 2, the even/odd blocks from N = 3 on).  A block takes NC cells, one
// column each (16 columns per row tile):
//   1. stages [cr W; cs W] and the face terms.  The velocity is constant, so a side's scaled flux is
//      A q- + B q+ with A = fscale (v.n + |v|), B = fscale (v.n - |v|) per cell face (AdvInst::coef): two
//      FP64 instructions on the trace values, read from W in place.  Each side forms its own flux;
//      a face kernel's flux array (a write and a read of 3 Nfp values per cell and stage) and its
//      launch are not needed, at the price of reading W of one buffer and writing another.
//   2. operand pre-pass, contraction, 3. recombination and the RK4 combine of advec_elem_kernel.
// 121-134 FP64 instructions per cell at N = 4 (116-127 us of the 256-261 us stage at K = 524288); the rest is the
// integer work of the exact product.  Step at K = 524288, N = 1 / 2 / 3 / 4: 404 / 800 / 1083 / 2449 ->
// 283 / 461 / 716 / 1039 us; K = 259200, N = 5 / 6: 1960 / 3093 -> 952 / 1231 us (before: a face kernel and
// an element kernel in FP64, on the tensor cores at N = 3).
template <int N>
constexpr size_t advec_fused_smem(int NC) {
  return (size_t)(nk_of(N) + np_of(N)) * (NC + 2) * sizeof(double) + NC * sizeof(int);
}
constexpr int advec_fused_threads(int NC) { return NC == 16 ? 128 : 256; }

template <int N, int NC>
__global__ void __launch_bounds__(advec_fused_threads(NC), 768 / advec_fused_threads(NC))
    advec_fused_kernel(const AdvInst d, const int stage, const double *__restrict__ in, double *__restrict__ out) {
  constexpr int Np = np_of(N), Nfp = N + 1, NF = 3 * Nfp, NK = nk_of(N), XS = NC + 2;
  constexpr int NUe = Sym<N>::NUe, NUo = Sym<N>::NUo, NRe = Sym<N>::NRe, NRo = Sym<N>::NRo;
  constexpr bool DENSE = N <= 2;
  constexpr int T = advec_fused_threads(NC);
  extern __shared__ __align__(16) double Xf[];  // [NK][XS]: slot, cell
  double *Y = Xf + NK * XS;                      // [Np][XS]: rows, cell
  int *Ems = reinterpret_cast<int *>(Y + Np * XS);
  __shared__ int s_pos[NK], s_fm[NF], s_out[Np];  // staging slots, face nodes, recombination
  const int t = threadIdx.x, e0 = blockIdx.x * NC, nc = min(NC, d.K - e0);
  for (int k = t; k < NK; k += T) s_pos[k] = (DENSE ? k : c_pos[N][k]) * XS;
  for (int k = t; k < NF; k += T) s_fm[k] = d.fmask[k];
  for (int k = t; k < Np; k += T)  // even row, odd row + 1 (0: none), sign
    s_out[k] = c_out[N][3 * k] | ((c_out[N][3 * k + 1] + 1) << 8) | (c_out[N][3 * k + 2] > 0 ? 1 << 16 : 0);
  __syncthreads();
  const size_t base = (size_t)e0 * Np;
  for (int j = t; j < NC * Np; j += T) {
    const int el = j / Np, k = j - el * Np;
    double2 c = make_double2(0.0, 0.0);
    double w = 0.0;
    if (el < nc) {
      c = ld2(d.coef + (size_t)(e0 + el) * 8);
      w = in[base + j];
    }
    Xf[s_pos[k] + el] = c.x * w;
    Xf[s_pos[Np + k] + el] = c.y * w;
  }
  for (int j = t; j < NC * NF; j += T) {
    const int el = j / NF, f = j - el * NF, fc = f / Nfp, i = f - fc * Nfp;
    double v = 0.0;
    if (el < nc) {
      const size_t e = e0 + el;
      const int2 nb = __ldg(&d.nbr[3 * e + fc]);  // {cell or -1, face | reverse << 2}
      const double2 c = ld2(d.coef + e * 8 + 2 + 2 * fc);
      const double qm = in[e * Np + s_fm[f]];
      const int ir = (nb.y >> 2) ? Nfp - 1 - i : i;
      const double qp = nb.x < 0 ? kAdvecGhost : in[(size_t)nb.x * Np + s_fm[(nb.y & 3) * Nfp + ir]];
      v = fma(c.x, qm, c.y * qp);
    }
    Xf[s_pos[2 * Np + f] + el] = v;
  }
  __syncthreads();
  const int lane = t & 31, warp = t >> 5;
  if constexpr (DENSE) {
    oz_product<N, 2, NK, Np, 0, 0, NK, Np, false, XS, NC / 16>(Xf, Y, warp, T / 32, lane);
  } else {
    oz_prep<NUe, NUo, XS, NC, T / NC>(Xf, Ems, t);
    __syncthreads();
    oz_product<N, 0, NUe, NRe, NUo, NRo, NUe, NRe, true, XS, NC / 16>(Xf, Y, warp, T / 32, lane, Ems);
  }
  __syncthreads();
  for (int j = t; j < nc * Np; j += T) {
    const int el = j / Np, i = j - el * Np;
    double r;
    if constexpr (DENSE) {
      r = Y[i * XS + el];
    } else {
      const int o = s_out[i], ro = ((o >> 8) & 0xFF) - 1;
      r = Y[(o & 0xFF) * XS + el];
      if (ro >= 0) r = (o >> 16) ? r + Y[ro * XS + el] : r - Y[ro * XS + el];
    }
    const size_t o = base + j;
    if (stage == 4) {
      d.rhs_out[o] = r;
      continue;
    }
    const double q = d.q[o], dt = d.dt;
    if (stage == 0) {
      d.acc[o] = r;
      out[o] = __dadd_rn(q, __dmul_rn(dt * 0.5, r));
    } else if (stage < 3) {
      d.acc[o] = __dadd_rn(d.acc[o], 2.0 * r);
      out[o] = __dadd_rn(q, __dmul_rn(stage == 1 ? dt * 0.5 : dt, r));
    } else {
      const double qn = __dadd_rn(q, __dmul_rn((1.0 / 6.0) * dt, __dadd_rn(d.acc[o], r)));
      d.q[o] = qn;
      out[o] = qn;
    }
  }
}

// The coefficients of AdvInst::coef for each cell: cr, cs, then (A, B) of faces 0..2.
__global__ void advec_coef_kernel(const AdvInst d, double *coef) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.K) return;
  const double *g = d.geo + (size_t)e * 16;
  double *c = coef + (size_t)e * 8;
  c[0] = d.vx * g[0] + d.vy * g[1];
  c[1] = d.vx * g[2] + d.vy * g[3];
  for (int f = 0; f < 3; f++) {
    const double vn = d.vx * g[4 + 3 * f] + d.vy * g[5 + 3 * f], fs = g[6 + 3 * f];
    c[2 + 2 * f] = fs * (vn + d.speed);
    c[3 + 2 * f] = fs * (vn - d.speed);
  }
}

// AdvInst::nbr from the edge records, a thread per edge; every cell face has exactly one edge
// (validate), so every entry is written once.  (Built on the host and copied, set-up took 2 ms more at
// K = 524288.)
__global__ void advec_nbr_kernel(const AdvInst d, int2 *nbr) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < d.nE) {
    const int4 e = d.edges[k];
    const int fL = e.z & 3, fR = (e.z >> 2) & 3, rev = (e.z >> 4) & 1;
    nbr[3 * (size_t)e.x + fL] = make_int2(e.y, fR | (rev << 2));
    nbr[3 * (size_t)e.y + fR] = make_int2(e.x, fL | (rev << 2));
  } else if (k - d.nE < d.nB) {
    const int4 b = d.bedges[k - d.nE];
    nbr[3 * (size_t)b.x + b.y] = make_int2(-1, 0);
  }
}

// advec/src/set_ic.h:3-10 at the node positions of src/init_grid.h.
template <int N>
__global__ void advec_ic_kernel(const AdvInst d, const double *coords, const int *cells) {
  constexpr int Np = np_of(N);
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (long long)d.K * Np) return;
  const int c = (int)(tid / Np), i = (int)(tid - (long long)c * Np);
  const int a = cells[3 * c], b = cells[3 * c + 1], e = cells[3 * c + 2];
  const double r = c_rs[N][i], s = c_rs[N][Np + i];
  const double x = node_coord(coords[2 * a], coords[2 * b], coords[2 * e], r, s);
  const double y = node_coord(coords[2 * a + 1], coords[2 * b + 1], coords[2 * e + 1], r, s);
  const double dx = __dsub_rn(x, 0.5), dy = __dsub_rn(y, 0.5);
  const double q = __dmul_rn(exp(__dmul_rn(__dmul_rn(-40.0, dx), dx)), exp(__dmul_rn(__dmul_rn(-40.0, dy), dy)));
  d.q[tid] = q;
  d.W[tid] = q;
}

// advec/src/save_solution.cpp:13-52: q at local nodes 0, N, Np-1 of the winning cell.
template <int N>
__global__ void advec_vertex_kernel(int K, const int *cells, const int *owner, const double *q, double *out) {
  constexpr int Np = np_of(N);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= K) return;
  const int local[3] = {0, N, Np - 1};
  for (int k = 0; k < 3; k++) {
    const int node = cells[3 * c + k];
    if (owner[node] == c) out[node] = q[(size_t)c * Np + local[k]];
  }
}

// Element-kernel forms 2 and 3, and at every order but 3 form 1, run advec_fused_kernel; form 1 at
// N = 3 the face kernel and the even/odd FP64 kernel, form 0 the face kernel and the dense one.
static bool advec_fused(int N) { return elem_form() >= (N == 3 ? 2 : 1); }

template <int N>
static void advec_launch_elem(const AdvInst &d, int stage, cudaStream_t s) {
  if constexpr (N == 3) {
    if (elem_form()) {
      advec_elem_kernel_sym<N><<<(d.K + 31) / 32, 32 * np_of(N), 0, s>>>(d, stage);
      return;
    }
  }
  advec_elem_kernel<N><<<(d.K + 31) / 32, 32 * np_of(N), 0, s>>>(d, stage);
}

// Stages 0..2 write the buffer that they do not read (W and W2 in turn), so that W holds the state
// after a step as before; the right-hand side alone (4) writes neither.
template <int N>
static void advec_launch_fused(const AdvInst &d, int stage, cudaStream_t s) {
  const double *in = (stage == 1 || stage == 3) ? d.W2 : d.W;
  double *out = (stage == 0 || stage == 2) ? d.W2 : d.W;
  auto go = [&](auto nc) {
    constexpr int NC = decltype(nc)::value;
    advec_fused_kernel<N, NC><<<(d.K + NC - 1) / NC, advec_fused_threads(NC), advec_fused_smem<N>(NC), s>>>(d, stage, in, out);
  };
  // Few cells: blocks of 16 (one row tile) spread them over the SMs.  Step, 16 / 128 cells a block:
  // K = 1152 24.8 / 47.1 us (N = 3), 29.9 / 69.4 (N = 4); K = 8192 29.6 / 49.0, 39.9 / 71.4; K = 16200
  // 55.4 / 49.7, 70.3 / 72.4; K = 32768 79.8 / 63.3, 107.3 / 91.4 us.
  if (d.K <= 12288) go(std::integral_constant<int, 16>());
  else go(std::integral_constant<int, 128>());
}

template <int N>
static void advec_launch_face(const AdvInst &d, cudaStream_t s) {
  const int nf = (d.nE + d.nB) * (N + 1);
  if (nf) advec_face_kernel<N><<<(nf + 255) / 256, 256, 0, s>>>(d);
}

template <int N>
static void advec_launch_stage(const AdvInst &d, int stage, cudaStream_t s) {
  if (advec_fused(N)) {
    advec_launch_fused<N>(d, stage, s);
  } else {
    advec_launch_face<N>(d, s);
    advec_launch_elem<N>(d, stage, s);
  }
}

Advection::~Advection() {
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  if (graph) cudaGraphDestroy(graph);
  if (graphG_exec) cudaGraphExecDestroy(graphG_exec);
  if (graphG) cudaGraphDestroy(graphG);
  for (void *p : allocs) cudaFree(p);
  if (stream) cudaStreamDestroy(stream);
}

int Advection::create(const Mesh &m, int order, double vel_x, double vel_y, double dt, std::string &err) {
  if (int rc = validate(m, err)) return rc;
  if (int rc = load_order_constants(order, err)) return rc;
  if (!(dt > 0.0) || !std::isfinite(dt) || !std::isfinite(vel_x) || !std::isfinite(vel_y)) {
    err = "dt must be positive and the velocity finite";
    return -4;
  }
  CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  N = order;
  K = m.n_cells();
  const int Np = np_of(N), Nfp = N + 1;
  Operators o;
  build_operators(N, o);
  d = AdvInst();
  d.N = N;
  d.K = K;
  d.nE = m.n_edges();
  d.nB = m.n_bedges();
  d.vx = vel_x;
  d.vy = vel_y;
  d.speed = std::sqrt(vel_x * vel_x + vel_y * vel_y);  // advec/src/advec_rhs.h:57
  d.dt = dt;
  std::vector<int4> edges, bedges;
  edge_records(m, edges, bedges);
  auto alloc = [&](size_t bytes) {
    void *p = nullptr;
    if (cudaMalloc(&p, bytes ? bytes : 16) != cudaSuccess) return (void *)nullptr;
    allocs.push_back(p);
    return p;
  };
  const size_t nq = (size_t)K * Np;
  d.q = (double *)alloc(nq * 8);
  d.W = (double *)alloc(nq * 8);
  d.W2 = (double *)alloc(nq * 8);
  d.acc = (double *)alloc(nq * 8);
  d.flux = (double *)alloc((size_t)K * 3 * Nfp * 8);
  double *geo = (double *)alloc((size_t)K * 16 * 8);
  d.geo = geo;
  double *coef = (double *)alloc((size_t)K * 8 * 8);
  d.coef = coef;
  int2 *nbr = (int2 *)alloc((size_t)K * 3 * sizeof(int2));
  d.nbr = nbr;
  int4 *de = (int4 *)alloc(sizeof(int4) * d.nE), *db = (int4 *)alloc(sizeof(int4) * d.nB);
  d.edges = de;
  d.bedges = db;
  int *fm = (int *)alloc(sizeof(int) * 3 * Nfp);
  d.fmask = fm;
  coords_d = (double *)alloc(m.coords.size() * 8);
  cells_d = (int *)alloc(m.cell2nodes.size() * 4);
  for (void *p : {(void *)d.q, (void *)d.W, (void *)d.W2, (void *)d.acc, (void *)d.flux, (void *)geo, (void *)coef,
                  (void *)nbr, (void *)de, (void *)db,
                  (void *)fm, (void *)coords_d, (void *)cells_d})
    if (!p) { err = "cudaMalloc failed"; return -101; }
  CK(cudaMemcpyAsync(de, edges.data(), sizeof(int4) * d.nE, cudaMemcpyHostToDevice, stream));
  CK(cudaMemcpyAsync(db, bedges.data(), sizeof(int4) * d.nB, cudaMemcpyHostToDevice, stream));
  CK(cudaMemcpyAsync(fm, o.FMASK.data(), sizeof(int) * 3 * Nfp, cudaMemcpyHostToDevice, stream));
  CK(cudaMemcpyAsync(coords_d, m.coords.data(), m.coords.size() * 8, cudaMemcpyHostToDevice, stream));
  CK(cudaMemcpyAsync(cells_d, m.cell2nodes.data(), m.cell2nodes.size() * 4, cudaMemcpyHostToDevice, stream));
  CK(cudaMemsetAsync(d.flux, 0, (size_t)K * 3 * Nfp * 8, stream));
  CK(cudaMemsetAsync(d.acc, 0, nq * 8, stream));
  geometry_kernel<<<(K + 127) / 128, 128, 0, stream>>>(K, coords_d, cells_d, geo);
  advec_coef_kernel<<<(K + 127) / 128, 128, 0, stream>>>(d, coef);
  advec_nbr_kernel<<<(d.nE + d.nB + 127) / 128, 128, 0, stream>>>(d, nbr);
  CK(cudaGetLastError());
  DG_DISPATCH(N, CK(cudaFuncSetAttribute(advec_fused_kernel<NN, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)advec_fused_smem<NN>(128))));  // 16 cells need 16 KB at most
  CK(cudaStreamSynchronize(stream));
  return 0;
}

int Advection::init(std::string &err) {
  const long long n = (long long)K * np_of(N);
  DG_DISPATCH(N, (advec_ic_kernel<NN><<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(d, coords_d, cells_d)));
  CK(cudaGetLastError());
  t = 0.0;
  steps = 0;
  return 0;
}

void Advection::enqueue_step(cudaStream_t s) {
  DG_DISPATCH(N, (advec_launch_stage<NN>(d, 0, s), advec_launch_stage<NN>(d, 1, s),
                  advec_launch_stage<NN>(d, 2, s), advec_launch_stage<NN>(d, 3, s)));
}

void Advection::enqueue_step_events(cudaStream_t s, cudaEvent_t *ev) {
  for (int stage = 0; stage < 4; stage++) {
    if (!advec_fused(N)) DG_DISPATCH(N, advec_launch_face<NN>(d, s));
    cudaEventRecord(ev[1 + 2 * stage], s);
    if (advec_fused(N)) {
      DG_DISPATCH(N, advec_launch_fused<NN>(d, stage, s));
    } else {
      DG_DISPATCH(N, advec_launch_elem<NN>(d, stage, s));
    }
    cudaEventRecord(ev[2 + 2 * stage], s);
  }
}

int Advection::step(int nsteps, bool use_graph, std::string &err) {
  auto capture = [&](int G, cudaGraph_t &g, cudaGraphExec_t &ex) -> int {
    if (ex) return 0;
    if (!graph_exec && !graphG_exec) set = launch_set_now();  // for both graphs
    const UseLaunchSet use(set);
    CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < G; k++) enqueue_step(stream);
    cudaError_t ce = cudaStreamEndCapture(stream, &g);
    if (ce != cudaSuccess) { err = std::string("graph capture: ") + cudaGetErrorString(ce); return -6; }
    CK(cudaGraphInstantiate(&ex, g, 0));
    return 0;
  };
  int i = 0;
  if (use_graph && nsteps >= kGraphSteps) {
    if (int rc = capture(kGraphSteps, graphG, graphG_exec)) return rc;
    for (; i + kGraphSteps <= nsteps; i += kGraphSteps) CK(cudaGraphLaunch(graphG_exec, stream));
  }
  if (use_graph && i < nsteps)
    if (int rc = capture(1, graph, graph_exec)) return rc;
  for (; i < nsteps; i++) {
    if (use_graph) CK(cudaGraphLaunch(graph_exec, stream));
    else enqueue_step(stream);
  }
  CK(cudaGetLastError());
  for (int k = 0; k < nsteps; k++) t += d.dt;  // advec/src/advec.cpp:262
  steps += (unsigned long long)nsteps;
  return 0;
}

int Advection::rhs(double *out_dev, std::string &err) {
  AdvInst r = d;
  r.rhs_out = out_dev;
  DG_DISPATCH(N, (advec_launch_stage<NN>(r, 4, stream)));
  CK(cudaGetLastError());
  return 0;
}

int Advection::vertex_values(int n_nodes, double *out_host, std::string &err) {
  int *owner = nullptr;
  double *buf = nullptr;
  CK(cudaMallocAsync((void **)&owner, (size_t)n_nodes * 4, stream));
  CK(cudaMallocAsync((void **)&buf, (size_t)n_nodes * 8, stream));
  CK(cudaMemsetAsync(owner, 0xff, (size_t)n_nodes * 4, stream));
  CK(cudaMemsetAsync(buf, 0, (size_t)n_nodes * 8, stream));
  vertex_owner_kernel<<<(K + 127) / 128, 128, 0, stream>>>(K, cells_d, owner);
  DG_DISPATCH(N, (advec_vertex_kernel<NN><<<(K + 127) / 128, 128, 0, stream>>>(K, cells_d, owner, d.q, buf)));
  CK(cudaMemcpyAsync(out_host, buf, (size_t)n_nodes * 8, cudaMemcpyDeviceToHost, stream));
  CK(cudaFreeAsync(owner, stream));
  CK(cudaFreeAsync(buf, stream));
  CK(cudaStreamSynchronize(stream));
  return 0;
}

}  // namespace dg
