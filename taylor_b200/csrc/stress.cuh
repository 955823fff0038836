// stress.cuh -- the stress update of one node (FINT.F90:363-870, 999-1116):
// shared by the kernels with a thread per node (force.cu) and the row gather
// that goes on to it (tiled.cu).
#pragma once
#include "mega_internal.cuh"

namespace mega {
namespace {

__device__ __forceinline__ NodeMat to_nodemat(const MatEntry& e) {
  NodeMat m;
  m.type = e.type; m.nu = e.nu; m.E = e.E; m.rho = e.rho; m.sig0 = e.sig0; m.B = e.B; m.C = e.C;
  m.lam = e.lam; m.mu = e.mu; m.l2m = e.l2m; m.p7 = e.p7; m.p8 = e.p8;
  return m;
}

template <typename T>
__device__ __forceinline__ T block_sum(T v, T* sm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sm[wid] = v;
  __syncthreads();
  T r = T(0);
  if (wid == 0) {
    r = (lane < (int)(blockDim.x >> 5)) ? sm[lane] : T(0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  }
  return r;  // valid in thread 0
}

// State of one node between the trial part of the update (kinematics,
// rotation, elastic predictor) and the rest (return mapping, write-back).
// LEAN: the old stress / strain and the material entry are re-read by the
// second part instead of held (the members stay unused and take no
// registers), which keeps the state small across the learned kernel's
// network evaluation.
template <typename T, bool LEAN>
struct Trial {
  double spred[6];
  T eps6[6], D[6], IF[3][3];
  double det;
  int mi;  // material table index
  double sold[6], eold[6];
  MatEntry me;
};

// FINT.F90:363-794: |det F|, INV3(F), L = G0 INV3(F), Hughes-Winget, rotation
// of sigma and eps, eps += dstrain, elastic predictor.
// DAM: the context holds damaged models (materials 3, 6) and their state;
// without it their branches compile out of the J2 path.
template <typename T, bool LEAN, bool DAM, bool FAST = false>
__device__ __forceinline__ void stress_trial(const StressArgs& a, int64_t i, Trial<T, LEAN>& w) {
  // F and G0 (18 planes), stress and strain (6 each) as 16-byte loads
  double fgi[18], sv[6], ev[6];
  load_fg(a.fg, fg_ld(a.n), i, sizeof(T) == 4, a.add_g0, fgi);
  {
    const double2* s2 = reinterpret_cast<const double2*>(a.stress + 6 * i);
    const double2* e2 = reinterpret_cast<const double2*>(a.strain + 6 * i);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double2 v = s2[k], u = e2[k];
      sv[2 * k] = v.x; sv[2 * k + 1] = v.y; ev[2 * k] = u.x; ev[2 * k + 1] = u.y;
    }
  }
  w.mi = a.matidx[i];
  if (!LEAN) w.me = a.mats[w.mi];
  const MatEntry& me = LEAN ? a.mats[w.mi] : w.me;
  T G0[3][3], L[3][3], sig[6], dstr[6];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int l = 0; l < 3; ++l) G0[k][l] = (T)fgi[9 + 3 * k + l];
  w.det = 1.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double so = sv[k], eo = ev[k];
    if (!LEAN) { w.sold[k] = so; w.eold[k] = eo; }
    sig[k] = (T)so;
    w.eps6[k] = (T)eo;
    w.D[k] = T(0);
  }
  if (FAST || a.finite_strain) {
    // |det F| and INV3 in double (F carries the FP64 displacement path)
    double Fd[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) Fd[k][l] = fgi[3 * k + l];
    w.det = det_abs(Fd);
    double IFd[3][3];
    inv3(Fd, IFd, a.inv3_exact != 0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) w.IF[k][l] = (T)IFd[k][l];
    mm3(G0, w.IF, L);
    T R[3][3];
    hughes_winget(L, R, dstr, w.D, a.inv3_exact != 0);
    rotate_tensor(R, sig);
    rotate_tensor(R, w.eps6);
  } else {
    // FINT.F90:772-783 small strain: engineering shear, no rotation, DET = 1
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) w.IF[k][l] = (k == l) ? T(1) : T(0);
    dstr[0] = G0[0][0]; dstr[1] = G0[1][1]; dstr[2] = G0[2][2];
    dstr[3] = G0[2][1] + G0[1][2]; dstr[4] = G0[2][0] + G0[0][2]; dstr[5] = G0[1][0] + G0[0][1];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) w.eps6[k] = w.eps6[k] + dstr[k];
  // the damaged models predict in effective space: STRESS / (1 - DAM)
  // (CONSTITUTE_VONMISES_DAM.F90:83, CONSTITUTE_DRUCKPRAG.F90:79)
  if (DAM && damaged_type(me.type)) {
    const T keep = T(1) - (T)a.aux[4 * i + 2];
#pragma unroll
    for (int k = 0; k < 6; ++k) sig[k] = sig[k] / keep;
  }
  // elastic predictor with FORM_CMAT (FINT_FUNCTIONS.F90:252-288)
  const T lam = (T)me.lam, mu = (T)me.mu, l2m = (T)me.l2m;
  w.spred[0] = (double)(sig[0] + (l2m * dstr[0] + lam * dstr[1] + lam * dstr[2]));
  w.spred[1] = (double)(sig[1] + (lam * dstr[0] + l2m * dstr[1] + lam * dstr[2]));
  w.spred[2] = (double)(sig[2] + (lam * dstr[0] + lam * dstr[1] + l2m * dstr[2]));
  w.spred[3] = (double)(sig[3] + mu * dstr[3]);
  w.spred[4] = (double)(sig[4] + mu * dstr[4]);
  w.spred[5] = (double)(sig[5] + mu * dstr[5]);
}

// Inputs of the surrogate network for a rate-dependent node: with q the
// trial deviatoric norm, sy0 = A + B eps0^n and f = q - sqrt(2/3) sy0,
//   x0 = ln(f / (sqrt(2/3) sy0))            overstress
//   x1 = eps0^n                             hardening state
//   x2 = ln(max(sqrt(2/3) f/(2 mu)/dt, epsdot0)/epsdot0) / 10   rate
//   x3 = 1e3 sqrt(2/3) sy0 / (2 mu)          yield-strain scale
// The target is y = dgamma / ub with ub = rate_upper_bound(f, eps0).
// Returns f (<= 0: elastic) and ub.
__device__ __forceinline__ double rate_features(const double spred[6], double eps0, const MatEntry& me, double dt,
                                                float x[4], double& ub) {
  const double mu = me.E / (2.0 * (1.0 + me.nu));
  const double kk = spred[0] + spred[1] + spred[2];
  const double d0 = spred[0] - kk / 3.0, d1 = spred[1] - kk / 3.0, d2 = spred[2] - kk / 3.0;
  const double q = sqrt(d0 * d0 + d1 * d1 + d2 * d2 + 2.0 * (spred[3] * spred[3] + spred[4] * spred[4] +
                                                             spred[5] * spred[5]));
  const double s23 = sqrt(2.0 / 3.0);
  const double epn = (eps0 > 0.0) ? pow(eps0, me.C) : 0.0;
  const double sy0 = me.sig0 + me.B * epn;
  const double f = q - s23 * sy0;
  const double dgpp = f / (2.0 * mu);
  ub = f > 0.0 ? rate_upper_bound(f, eps0, mu, me.B, me.C) : 0.0;
  x[0] = (float)log(fmax(f, 1e-30 * sy0) / (s23 * sy0));
  x[1] = (float)epn;
  x[2] = (float)(log(fmax(s23 * dgpp / dt, me.p8) / me.p8) / 10.0);
  x[3] = (float)(1e3 * s23 * sy0 / (2.0 * mu));
  return f;
}

// FINT.F90:797-870, 999-1116: return mapping (dg0 >= 0 starts the rate law's
// Newton there), state write-back, strain_eq, internal work, wave speed, T_i.
template <typename T, typename TS, bool LEAN, bool DAM, bool FAST = false>
__device__ __forceinline__ void stress_finish(const StressArgs& a, int64_t i, Trial<T, LEAN>& w, double dg0, double& work,
                                              unsigned long long& nit, unsigned long long& npl, unsigned& st) {
  const MatEntry& me = LEAN ? a.mats[w.mi] : w.me;
  const NodeMat m = to_nodemat(me);
  const double vol = a.vol[i];
  double snew[6];
  double ep = a.eps[i];
  const double ep0 = ep;
  int it = 0;
  bool cap = false;
  if (m.type == MEGA_MAT_ELASTIC) {
#pragma unroll
    for (int k = 0; k < 6; ++k) snew[k] = w.spred[k];
  } else if (m.type == MEGA_MAT_VONMISES) {
    it = von_mises(w.spred, ep, m, a.maxit, snew, cap);
  } else if (m.type == MEGA_MAT_VM_RATE) {
    double dg = 0.0, ftr = 0.0;
    const double dt = a.ndt ? a.ndt[i] : a.dt;
    it = vm_rate(w.spred, ep, m, dt, a.rtol, a.maxit, a.rate_solver, dg0, snew, cap, dg, ftr);
    if (a.log_buf && it > 0) {  // sample (features, converged multiplier) for the surrogate
      const uint64_t sb = (uint64_t)__double_as_longlong(w.spred[0]);
      const uint32_t hsh = ((uint32_t)i * 2654435761u) ^ (uint32_t)(sb ^ (sb >> 29)) ^ a.log_seed;
      if (hsh % a.log_stride == 0) {
        float x[4];
        double ub;
        const double f = rate_features(w.spred, ep0, me, dt, x, ub);
        if (f > 0.0 && ub > 0.0) {
          const unsigned long long k = atomicAdd(a.log_count, 1ull);
          if ((int64_t)k < a.log_cap) {
            float* o = a.log_buf + 5 * k;
            o[0] = x[0]; o[1] = x[1]; o[2] = x[2]; o[3] = x[3];
            o[4] = (float)(dg / ub);
          }
        }
      }
    }
  } else if (DAM && damaged_type(m.type)) {
    // CONSTITUTION.F90:60-64, 72-76: the total strain (already advanced by
    // dstrain) and the four damage-state values ride along; spred is the
    // effective predictor
    double tot[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) tot[k] = (double)w.eps6[k];
    double2* a2 = reinterpret_cast<double2*>(a.aux + 4 * i);
    const double2 x0 = a2[0], x1 = a2[1];
    double ax[4] = {x0.x, x0.y, x1.x, x1.y};
    const DamageMat d{me.ki, me.kc, me.dmax, me.qphi, me.kphi, me.qpsi};
    if (m.type == MEGA_MAT_VM_DAMAGE) it = von_mises_dam(w.spred, tot, ep, ax, m, d, a.maxit, snew, cap);
    else it = drucker_prager(w.spred, tot, ep, ax, m, d, snew);
    a2[0] = make_double2(ax[0], ax[1]);
    a2[1] = make_double2(ax[2], ax[3]);
  } else {
    st |= MEGA_ST_BAD_MATERIAL;
#pragma unroll
    for (int k = 0; k < 6; ++k) snew[k] = w.spred[k];
  }
  if (cap) st |= MEGA_ST_NEWTON_CAP;
  nit += (unsigned long long)it;
  npl += (it > 0) ? 1ull : 0ull;
  if (!FAST && a.iters && !a.more) a.iters[i] = it;
  double sinc[6], einc[6], enew[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    enew[k] = (double)w.eps6[k];
    sinc[k] = snew[k] - (LEAN ? a.stress[6 * i + k] : w.sold[k]);
    einc[k] = enew[k] - (LEAN ? a.strain[6 * i + k] : w.eold[k]);
  }
  if (a.stress_prev) {
    double2* p2 = reinterpret_cast<double2*>(a.stress_prev + 6 * i);
    const double2* old = reinterpret_cast<const double2*>(a.stress + 6 * i);
#pragma unroll
    for (int k = 0; k < 3; ++k) p2[k] = LEAN ? old[k] : make_double2(w.sold[2 * k], w.sold[2 * k + 1]);
  }
  {
    double2* s2 = reinterpret_cast<double2*>(a.stress + 6 * i);
    double2* e2 = reinterpret_cast<double2*>(a.strain + 6 * i);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s2[k] = make_double2(snew[2 * k], snew[2 * k + 1]);
      e2[k] = make_double2(enew[2 * k], enew[2 * k + 1]);
    }
  }
  a.eps[i] = ep;
  if (FAST || a.finite_strain) {
#pragma unroll
    for (int k = 0; k < 6; ++k) work += 0.5 * (double)w.D[k] * (2.0 * snew[k] - sinc[k]) * vol * w.det;
  } else {
#pragma unroll
    for (int k = 0; k < 6; ++k) work += 0.5 * einc[k] * sinc[k] * vol * w.det;
  }
  if (!FAST && !a.more) {  // the last step of a call: what only a caller reads
    const double eq = enew[0] * enew[0] + enew[1] * enew[1] + enew[2] * enew[2] +
                      2.0 * (enew[3] * enew[3] + enew[4] * enew[4] + enew[5] * enew[5]);
    a.strain_eq[i] = sqrt(eq * 2.0 / 3.0);
    double bulk = m.E / (3.0 * (1.0 - 2.0 * m.nu)), shear = m.E / (2.0 * (1.0 + m.nu));
    if (m.type > 1) estimate_moduli(sinc, einc, shear, bulk);
    const double pmod = bulk + 4.0 * shear / 3.0;
    a.wvel[i] = sqrt(fmax(pmod, shear) / m.rho);
  }
  // T_i = V J sigma IF^T: f_J(k) = sum_m T(k,m) grad0 phi_iJ(m)
  const T vj = (T)(vol * w.det);
  T S[3][3];
  T sn[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) sn[k] = (T)snew[k];
  v2t(sn, S);
  TS tv[12];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int mm = 0; mm < 3; ++mm)
      tv[3 * k + mm] = (TS)(vj * (S[k][0] * w.IF[mm][0] + S[k][1] * w.IF[mm][1] + S[k][2] * w.IF[mm][2]));
  tv[9] = tv[10] = tv[11] = TS(0);
  if (a.has_body) {
    const double rvj = m.rho * vol * w.det;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double b = (a.bodyforce ? a.bodyforce[3 * i + k] : 0.0) + a.grav[k];
      tv[9 + k] = (TS)(b * rvj);
    }
  }
  // the 12-value row (48 or 96 bytes, 16-byte aligned) as vector stores
  if (sizeof(TS) == 4) {
    float4* t4 = reinterpret_cast<float4*>((TS*)a.tmat + 12 * i);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      t4[k] = make_float4((float)tv[4 * k], (float)tv[4 * k + 1], (float)tv[4 * k + 2], (float)tv[4 * k + 3]);
  } else {
    double2* t2 = reinterpret_cast<double2*>((TS*)a.tmat + 12 * i);
#pragma unroll
    for (int k = 0; k < 6; ++k) t2[k] = make_double2((double)tv[2 * k], (double)tv[2 * k + 1]);
  }
#pragma unroll
  for (int k = 0; k < 6; ++k)
    if (!isfinite(snew[k])) st |= MEGA_ST_NONFINITE;
}

// STEP: the counts of this step alone too (zeroed by the row gather before).
template <typename T, bool STEP = true>
__device__ __forceinline__ void stress_reduce(const StressArgs& a, double work, unsigned long long nit,
                                              unsigned long long npl, unsigned st, double* smd,
                                              unsigned long long* smu) {
  const double wsum = block_sum(work, smd);
  const unsigned long long it_sum = block_sum(nit, smu);
  const unsigned long long pl_sum = block_sum(npl, smu);
  if (threadIdx.x == 0) {
    const int sl = blockIdx.x % kSlots;
    if (wsum != 0.0) atomicAdd(&a.acc->int_work[sl], wsum);
    if (it_sum) {
      if (STEP) atomicAdd(&a.acc->newton_iters[sl], it_sum);
      atomicAdd(&a.acc->newton_total[sl], it_sum);
    }
    if (pl_sum) {
      if (STEP) atomicAdd(&a.acc->plastic[sl], pl_sum);
      atomicAdd(&a.acc->plastic_total[sl], pl_sum);
    }
  }
  if (st) atomicOr(a.status, st);
}

}  // namespace
}  // namespace mega
