// Implicit-shift QL / QR / root-free PWK iterations on the tridiagonal, one
// matrix per lane or per four lanes (matrices sorted by size so that those
// of a warp run similar-length loops).
//
// Replaces, per matrix:
//   eigQL!          (GenericLinearAlgebra.jl src/eigenSelfAdjoint.jl:221-288)
//   singleShiftQL!  (:377-409)
//   eigQR!          (:290-340), singleShiftQR! (:412-444)
//   eigvalsPWK!     (:163-219), singleShiftQLPWK! (:343-374)
//   eig2x2! / eigvals2x2 (:131-161)
//   givensAlgorithm for Float64/Float32 (LinearAlgebra's LAPACK-dlartg port).
//
// The scalar recurrence of a chase is serial. FP32 chases and the root-free
// one (k_chase) run one matrix per lane; FP64 QL and QR (k_chase_grp), four
// lanes per matrix: there an FP64 warp instruction costs its unit ~64 cycles
// whatever the active-lane count, and one of them does several products. The
// rotations (c, s) are not applied here: they are appended to a per-matrix
// log (plus one header per sweep) that the apply kernel replays on the rows
// of Q in parallel. When a matrix's log is full the lane stops between
// sweeps, saves its state and is resumed by the next pass.
//
// Differences from the reference, all rounding-level: the Givens radius
// uses a Newton-refined hardware rsqrt seed instead of sqrt and two
// divisions; gamma/c uses a refined reciprocal; the deflation test
// |e| <= tol*sqrt|d_i|*sqrt|d_i+1| (:250-256) is decided on exponents when
// the two sides are more than a factor 4 apart and evaluated exactly
// otherwise (identical decisions on identical data). Each chase is capped at
// max_sweeps_per_n * n sweeps (the reference has no cap and loops forever on
// e.g. NaN input); hitting the cap reports the unconverged count as info.
#include <algorithm>

#include "gla_launch.h"
#include "gla_small.cuh"

namespace gla {

template <class T> GLA_DEV bool is_zero(T x) { return (prec<T>::bits(x) << 1) == 0; }

// Deflation test of :250-256 (and of :177 with e holding e^2) on the exponents
// alone: 1 negligible, 0 not, 2 undecided.
template <class T> GLA_DEV int negligible_fast(T ev, T d1, T d2, int tol_e) {
  const unsigned maxe = sizeof(T) == 8 ? 0x7ff : 0xff;
  const int xe = prec<T>::biased_exp(ev), x1 = prec<T>::biased_exp(d1), x2 = prec<T>::biased_exp(d2);
  const bool normal = (unsigned)xe - 1 < maxe - 1 && (unsigned)x1 - 1 < maxe - 1 && (unsigned)x2 - 1 < maxe - 1;
  // q = 2log2|e| - log2|d1| - log2|d2| - 2log2(tol) lies in (L-4, L+2)
  const int L = 2 * xe - x1 - x2 - 2 * tol_e;
  return !normal ? 2 : (L + 2 <= 0 ? 1 : (L - 4 >= 0 ? 0 : 2));
}
template <class T> GLA_DEV bool negligible(T ev, T d1, T d2, T tol, int tol_e) {
  const int f = negligible_fast(ev, d1, d2, tol_e);
  if (f != 2) return f != 0;
  return tabs(ev) <= tol * prec<T>::sqrt_ieee(tabs(d1)) * prec<T>::sqrt_ieee(tabs(d2));
}

// LAPACK 3.x dlartg convention (as in LinearAlgebra.givensAlgorithm for
// AbstractFloat): r = +-sqrt(f^2+g^2), (c,s,r) negated when |f|>|g| and c<0.
template <class T> GLA_DEV void givens_exact(T f, T g, T& cs, T& sn, T& r) {
  const T safmn2 = sizeof(T) == 8 ? (T)0x1p-485 : (T)0x1p-51f;
  const T safmx2 = T(1) / safmn2;
  T f1 = f, g1 = g;
  T scale = fmax(tabs(f1), tabs(g1));
  int count = 0;
  if (scale >= safmx2) {
    do {
      count++;
      f1 *= safmn2;
      g1 *= safmn2;
      scale = fmax(tabs(f1), tabs(g1));
    } while (scale >= safmx2 && count < 20);
    r = prec<T>::sqrt_ieee(f1 * f1 + g1 * g1);
    cs = prec<T>::div_ieee(f1, r);
    sn = prec<T>::div_ieee(g1, r);
    for (int i = 0; i < count; i++) r *= safmx2;
  } else if (scale <= safmn2) {
    do {
      count++;
      f1 *= safmx2;
      g1 *= safmx2;
      scale = fmax(tabs(f1), tabs(g1));
    } while (scale <= safmn2 && count < 4000);
    r = prec<T>::sqrt_ieee(f1 * f1 + g1 * g1);
    cs = prec<T>::div_ieee(f1, r);
    sn = prec<T>::div_ieee(g1, r);
    for (int i = 0; i < count; i++) r *= safmn2;
  } else {
    r = prec<T>::sqrt_ieee(f1 * f1 + g1 * g1);
    cs = prec<T>::div_ieee(f1, r);
    sn = prec<T>::div_ieee(g1, r);
  }
}

template <class T> GLA_DEV void givens(T f, T g, T& c, T& s, T& r) {
  if (is_zero(g)) {
    c = 1;
    s = 0;
    r = f;
    return;
  }
  if (is_zero(f)) {
    c = 0;
    s = 1;
    r = g;
    return;
  }
  if (prec<T>::squares(f) && prec<T>::squares(g)) {
    const T r2 = fma(f, f, g * g);
    const T y = prec<T>::rsqrt(r2);
    r = r2 * y;
    c = f * y;
    s = g * y;
  } else {
    givens_exact(f, g, c, s, r);
  }
  // |f| > |g| and c < 0 (c has the sign of f)
  if (!abs_le(f, g) && (prec<T>::bits(c) >> (sizeof(T) * 8 - 1))) {
    c = -c;
    s = -s;
    r = -r;
  }
}

// Givens rotation for the FP32 sweep step: the refined-rsqrt radius when
// f^2 + g^2 is comfortably inside the normal range, the exact dlartg port
// otherwise. Same convention as givens() (c >= 0 when |f| > |g|; f == 0 gives
// c = 0, s = 1, r = g).
GLA_DEV void givens_step(float f, float g, float& c, float& s, float& r) {
  const float r2 = fmaf(f, f, g * g);
  if (r2 >= 0x1p-120f && r2 <= 0x1p+120f) {
    const float y = prec<float>::rsqrt(r2);
    r = r2 * y;
    c = f * y;
    s = g * y;
    if (f == 0.f) {
      c = 0.f;
      s = 1.f;
      r = g;
    } else if (f < 0.f && fabsf(f) > fabsf(g)) {
      c = -c;
      s = -s;
      r = -r;
    }
  } else {
    givens(f, g, c, s, r);
  }
}

// Deflation test on register values: FP32 decides on the squared sides
// (margin 4x each way) and falls back to the exact form near the threshold
// or when a square leaves the normal range; FP64 uses the exponent filter.
GLA_DEV bool negligible_step(float ev, float d1, float d2, float tol, int tol_e) {
  const float e2 = ev * ev;
  const float rhs = (tol * tol) * fabsf(d1 * d2);
  if (rhs >= 0x1p-120f && rhs <= 0x1p+120f && e2 <= 0x1p+120f) {
    if (e2 < 0.25f * rhs) return true;
    if (e2 > 4.f * rhs) return false;
  }
  return negligible(ev, d1, d2, tol, tol_e);
}
GLA_DEV bool negligible_step(double ev, double d1, double d2, double tol, int tol_e) {
  return negligible(ev, d1, d2, tol, tol_e);
}

// gamma / c: FP32 uses rcp.approx (~1 ulp, one rounding in the recurrence)
// guarded by a float compare; FP64 the Newton-refined reciprocal.
GLA_DEV float div_step(float a, float b) {
  if (fabsf(b) < 0x1p-100f) return __fdiv_rn(a, b);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return a * y;
}

template <class T> GLA_DEV T div_fast(T a, T b) {
  return prec<T>::tame(b) ? a * prec<T>::rcp(b) : prec<T>::div_ieee(a, b);
}

// Append (c, s) to the rotation log as one 8-byte store.
GLA_DEV void store_rot(float* log, int k, float c, float s) {
  reinterpret_cast<float2*>(log)[k] = make_float2(c, s);
}

// sqrt(m^2 + 1) for the shift computation (:272, :201, :325); exactness of
// the shift only affects the convergence rate, so a refined rsqrt replaces
// the correctly rounded hypot here.
template <class T> GLA_DEV T hypot1_fast(T m) {
  const T am = tabs(m);
  if (!prec<T>::squares(am)) return am < T(1) ? T(1) : am;
  const T q = fma(m, m, T(1));
  return q * prec<T>::rsqrt(q);
}

size_t chase_smem_bytes(int nmax, int elem) { return 512 + (size_t)2 * nmax * 32 * elem; }

// ALGO: kAlgoQL (eigQL!, logs rotations), kAlgoQR (eigQR!, logs), kAlgoPWK
// (eigvalsPWK!, values only). d, e: per-matrix diagonals at w_off (e padded
// to n entries). rot: 2 values per rotation; hdr: one word per sweep.
//
// Deflation bookkeeping: instead of rescanning e from blockstart after every
// chase (:250-256), each lane keeps a bitmask NF of "e[j] is negligible",
// re-evaluating entry j exactly when e[j], d[j] or d[j+1] takes its final
// value for the chase (one test per rotation). The first negligible entry at
// or after blockstart is then found with __ffs, and the decision is the one
// the rescan would make on the same values. This keeps the 32 lanes of a
// warp from serialising on each other's O(n) scans.
template <class T, int ALGO>
__global__ void __launch_bounds__(32) k_chase(const SmallDesc* __restrict__ descs, const int* __restrict__ perm,
                                              int count, T* __restrict__ dg_all, T* __restrict__ eg_all,
                                              ChaseState* __restrict__ cst, T* __restrict__ rot,
                                              unsigned* __restrict__ hdr, int* __restrict__ info, T tol,
                                              int max_sweeps_per_n, int* __restrict__ pending,
                                              unsigned long long* __restrict__ stats, int lanes_per_warp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x;
  // lanes_per_warp matrices per warp (the other lanes idle): fewer lanes cut
  // the divergence between lanes that are between sweeps and lanes inside one
  const int slot = blockIdx.x * lanes_per_warp + lane;
  const bool have = lane < lanes_per_warp && slot < count;
  const int mid = have ? perm[slot] : 0;
  SmallDesc dsc;
  dsc.n = 0;
  if (have) dsc = descs[mid];
  const int n = dsc.n;
  int nmax = n;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nmax = max(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
  unsigned* NF = reinterpret_cast<unsigned*>(smem_raw) + lane;  // NF[w * 32], w < 4
  T* D = reinterpret_cast<T*>(smem_raw + 512) + lane;
  T* E = reinterpret_cast<T*>(smem_raw + 512) + (size_t)nmax * 32 + lane;
#define DD(i) D[(size_t)(i) * 32]
#define EE(i) E[(size_t)(i) * 32]

  ChaseState st;
  st.status = kChaseDone;
  if (have) st = cst[mid];
  const bool was_running = have && st.status == kChaseRunning;
  bool active = was_running;
  T* dg = dg_all + dsc.w_off;
  T* eg = eg_all + dsc.w_off;
  const int tol_e = prec<T>::biased_exp(tol) - prec<T>::expbias;
  auto test = [&](int j) {  // re-evaluate NF(j), j <= n - 2
    const bool f = negligible(EE(j), DD(j), DD(j + 1), tol, tol_e);
    unsigned& w = NF[(j >> 5) * 32];
    const unsigned b = 1u << (j & 31);
    w = f ? (w | b) : (w & ~b);
  };
  auto first_nf = [&](int from) -> int {  // first j >= from with NF(j), else n - 1
    for (int w = from >> 5; w <= (n - 2) >> 5; w++) {
      unsigned bits = NF[w * 32];
      if (w == (from >> 5)) bits &= ~0u << (from & 31);
      if (bits) return w * 32 + __ffs(bits) - 1;
    }
    return n - 1;
  };
  for (int w = 0; w < 4; w++) NF[w * 32] = 0;
  if (active) {
    for (int k = 0; k < n; k++) {
      DD(k) = dg[k];
      const T e = eg[k];
      // eigvalsPWK! squares the off-diagonal first (:171-173)
      EE(k) = (ALGO == kAlgoPWK && st.nsweeps == 0 && st.bs == 0) ? e * e : e;
    }
    for (int j = 0; j + 1 < n; j++) test(j);
  }
  const int cap = max_sweeps_per_n * n;
  int bs = st.bs, nsw = st.nsweeps;
  int nrot = 0, nhdr = 0;
  T* myrot = rot + 2 * dsc.rot_off;
  unsigned* myhdr = hdr + dsc.hdr_off;
  bool insweep = false, stopped_full = false;
  int i = 0, be = 0;
  T mu = 0, gam = 0, p = 0, c = 1, s = 0;
  // register cache of the sweep: next (e, d) to consume, the d two positions
  // behind (for the deflation test) and e beyond the block end
  T e_nx = 0, d_nx = 0, d_up = 0, e_end = 0;
  // NF word of the current sweep position cached in a register
  unsigned nfw = 0;
  int nfw_idx = -1;
  auto nf_flush = [&]() {
    if (nfw_idx >= 0) NF[nfw_idx * 32] = nfw;
    nfw_idx = -1;
  };
  auto test_v = [&](int j, T ev, T d1, T d2) {  // NF(j) from register values
    const bool f = negligible_step(ev, d1, d2, tol, tol_e);
    const int wi = j >> 5;
    if (wi != nfw_idx) {
      nf_flush();
      nfw_idx = wi;
      nfw = NF[wi * 32];
    }
    const unsigned b = 1u << (j & 31);
    nfw = f ? (nfw | b) : (nfw & ~b);
  };
  int iters = 0;
  const int iter_cap = (max_sweeps_per_n + 4) * 4 * nmax * nmax + 64;  // hard bound on loop trips

  while (__any_sync(0xffffffffu, active)) {
    if (++iters > iter_cap) {  // defensive: never reached when the sweep cap works
      if (active) {
        info[mid] = max(1, n - 1);
        active = false;
        st.status = kChaseDone;
      }
      continue;
    }
    if (active && !insweep) {
      nf_flush();
      if (bs >= n - 1) {
        active = false;
        st.status = kChaseDone;
      } else {
        be = first_nf(bs);
        if (bs == be) {
          bs += 1;
        } else if (bs + 1 == be) {
          if (ALGO == kAlgoPWK) {
            const T d1 = DD(bs), d2 = DD(be), ee = prec<T>::sqrt_ieee(EE(bs));
            const T r1 = (d1 + d2) / 2;
            const T r2 = hypot_borges(d1 - d2, 2 * ee) / 2;
            DD(bs) = r1 + r2;
            DD(be) = r1 - r2;
            EE(bs) = 0;
            test(bs);
            if (be <= n - 2) test(be);
            bs += 1;
          } else if (nrot + 1 > dsc.rot_cap || nhdr + 1 > dsc.hdr_cap) {
            active = false;
            stopped_full = true;
          } else {
            // eig2x2! (:136-161)
            const T dj = DD(bs), dj1 = DD(be), ej = EE(bs);
            const T r1 = (dj + dj1) / 2;
            const T r2 = hypot_borges(dj - dj1, 2 * ej) / 2;
            const T lp = r1 + r2, lm = r1 - r2;
            DD(bs) = lp;
            DD(be) = lm;
            EE(bs) = 0;
            T cc, ss;
            if (is_zero(ej)) {
              cc = 1;
              ss = 0;
            } else if (tabs(lp - dj) > tabs(lm - dj)) {
              cc = prec<T>::div_ieee(-ej, hypot_borges(ej, lp - dj));
              ss = prec<T>::sqrt_ieee(1 - cc * cc);
            } else {
              ss = prec<T>::div_ieee(tabs(ej), hypot_borges(ej, lm - dj));
              cc = tcopysign(prec<T>::sqrt_ieee(1 - ss * ss), -ej);
            }
            myhdr[nhdr++] = pack_hdr(bs, 1, 0);
            myrot[2 * nrot] = cc;
            myrot[2 * nrot + 1] = ss;
            nrot++;
            test(bs);
            if (be <= n - 2) test(be);
            bs += 2;
          }
        } else if (nsw >= cap) {
          int cnt = 0;
          for (int b = 0; b + 1 < n; b++) cnt += !negligible(EE(b), DD(b), DD(b + 1), tol, tol_e);
          info[mid] = max(cnt, 1);
          active = false;
          st.status = kChaseDone;
        } else if (ALGO != kAlgoPWK && (nrot + (be - bs) > dsc.rot_cap || nhdr + 1 > dsc.hdr_cap)) {
          active = false;
          stopped_full = true;
        } else {
          // shift (:199-202 PWK, :271-273 QL, :324-326 QR) and start a chase
          if (ALGO == kAlgoPWK) {
            const T sqrte = prec<T>::sqrt_ieee(EE(bs));
            const T m = div_fast(DD(bs + 1) - DD(bs), 2 * sqrte);
            mu = DD(bs) - div_fast(sqrte, m + tcopysign(hypot1_fast(m), m));
            gam = DD(be) - mu;
            p = gam * gam;
            i = be - 1;
          } else if (ALGO == kAlgoQL) {
            const T m = div_fast(DD(bs + 1) - DD(bs), 2 * EE(bs));
            mu = DD(bs) - div_fast(EE(bs), m + tcopysign(hypot1_fast(m), m));
            gam = DD(be) - mu;
            p = gam;
            i = be - 1;
            myhdr[nhdr++] = pack_hdr(be - 1, be - bs, 0);
          } else {
            const T m = div_fast(DD(be - 1) - DD(be), 2 * EE(be - 1));
            mu = DD(be) - div_fast(EE(be - 1), m + tcopysign(hypot1_fast(m), m));
            gam = DD(bs) - mu;
            p = gam;
            i = bs + 1;
            myhdr[nhdr++] = pack_hdr(bs + 1, be - bs, 1);
          }
          if (ALGO == kAlgoQR) {
            e_nx = EE(bs);
            d_nx = DD(bs + 1);
            d_up = DD(bs);  // d[i-2] of the first test (unused: j < bs)
          } else {
            e_nx = EE(be - 1);
            d_nx = DD(be - 1);
            d_up = (be + 1 <= n - 1) ? DD(be + 1) : T(0);
            e_end = (be <= n - 2) ? EE(be) : T(0);
          }
          c = 1;
          s = 0;
          insweep = true;
          nsw++;
        }
      }
    }
    // tight sweep loop: runs while every active lane is inside a chase
    while (__all_sync(0xffffffffu, !active || insweep) && __any_sync(0xffffffffu, active)) {
      if (++iters > iter_cap) break;
      if (active) {
        if constexpr (ALGO == kAlgoQL) {
          // singleShiftQL! step at i (:389-405), operands from registers
          const T ei = e_nx, di = d_nx;
          if (i > bs) {
            e_nx = EE(i - 1);
            d_nx = DD(i - 1);
          }
          const T c1 = c, s1 = s;
          T zeta;
          givens_step(p, ei, c, s, zeta);
          const T enew = (i < be - 1) ? s1 * zeta : e_end;
          if (i < be - 1) EE(i + 1) = enew;
          const T g1 = gam;
          gam = c * c * (di - mu) - s * s * g1;
          const T dnew = g1 + di - gam;
          DD(i + 1) = dnew;
          p = is_zero(c) ? -ei * c1 : div_step(gam, c);
          store_rot(myrot, nrot, c, s);
          nrot++;
          if (i + 1 <= n - 2) test_v(i + 1, enew, dnew, d_up);
          d_up = dnew;
          i--;
          if (i < bs) {
            const T eb = s * p, db = mu + gam;
            EE(bs) = eb;
            DD(bs) = db;
            test_v(bs, eb, db, d_up);
            insweep = false;
          }
        } else if constexpr (ALGO == kAlgoQR) {
          // singleShiftQR! step at i (:424-440), operands from registers;
          // d_up holds d[i-2] (the previous step's new d)
          const T ei = e_nx, di = d_nx;
          if (i < be) {
            e_nx = EE(i);
            d_nx = DD(i + 1);
          }
          const T c1 = c, s1 = s;
          T zeta;
          givens_step(p, ei, c, s, zeta);
          const T g1 = gam;
          gam = c * c * (di - mu) - s * s * g1;
          const T dnew = g1 + di - gam;
          DD(i - 1) = dnew;
          if (i > bs + 1) {
            const T enew = s1 * zeta;
            EE(i - 2) = enew;
            test_v(i - 2, enew, d_up, dnew);
          }
          p = is_zero(c) ? -ei * c1 : div_step(gam, c);
          store_rot(myrot, nrot, c, s);
          nrot++;
          d_up = dnew;
          i++;
          if (i > be) {
            const T eb = s * p, db = mu + gam;
            EE(be - 1) = eb;
            DD(be) = db;
            test_v(be - 1, eb, d_up, db);
            if (be <= n - 2) test_v(be, EE(be), db, DD(be + 1));
            insweep = false;
          }
        } else {
          // singleShiftQLPWK! step at i (:356-370); e holds squares
          const T ei = e_nx, di = d_nx;
          if (i > bs) {
            e_nx = EE(i - 1);
            d_nx = DD(i - 1);
          }
          const T zeta = p + ei;
          const T enew = (i < be - 1) ? s * zeta : e_end;
          if (i < be - 1) EE(i + 1) = enew;
          const T c1 = c;
          const T rz = prec<T>::tame(zeta) ? prec<T>::rcp(zeta) : prec<T>::div_ieee(T(1), zeta);
          c = p * rz;
          s = ei * rz;
          const T g1 = gam;
          gam = c * (di - mu) - s * g1;
          const T dnew = g1 + di - gam;
          DD(i + 1) = dnew;
          p = is_zero(c) ? ei * c1 : div_fast(gam * gam, c);
          if (i + 1 <= n - 2) test_v(i + 1, enew, dnew, d_up);
          d_up = dnew;
          i--;
          if (i < bs) {
            const T eb = s * p, db = mu + gam;
            EE(bs) = eb;
            DD(bs) = db;
            test_v(bs, eb, db, d_up);
            insweep = false;
          }
        }
    
      }
    }
  }
  if (was_running) {
    for (int k = 0; k < n; k++) {
      dg[k] = DD(k);
      eg[k] = EE(k);
    }
    const int sweeps_this_pass = nsw - st.nsweeps;
    st.bs = bs;
    st.nsweeps = nsw;
    st.nrot = nrot;
    st.nhdr = nhdr;
    cst[mid] = st;
    if (stopped_full) atomicAdd(pending, 1);
    atomicAdd(&stats[0], (unsigned long long)(ALGO == kAlgoPWK ? 0 : nrot));
    atomicAdd(&stats[1], (unsigned long long)sweeps_this_pass);
    atomicAdd(&stats[2], (unsigned long long)(ALGO == kAlgoPWK ? 0 : nrot) * (unsigned long long)n);
  }
#undef DD
#undef EE
}

// ---------------------------------------------------------------- FP64 QL / QR: four lanes per matrix
//
// What bounds an FP64 chase is the number of FP64 warp instructions on its
// path: each one holds the sub-partition's unit for 64 cycles, whatever the
// lanes do with it, and its result is there when the unit is free again. So
// a matrix has a group of four lanes, and one instruction does up to four
// different products of its step (operands chosen per lane by 32-bit
// selects, results passed by shuffles of 24 cycles):
//
//   slot   lanes 0, 1              lane 2           lane 3
//   1      r2 = p p + ee           u = ee c1        gam = p c1
//   2      h  = r2 y0              nr = p a - u     d[i+1] = t - gam (last step's)
//   3      er = 1 - h y0           ee' = e' e'      t = gam + d_i
//   4      q = 3/8 er + 1/2 | y0 er  a' = d' - mu   e[i+1] = s r (last step's)
//   5      y = y0 + (y0 er) q      (all lanes)
//   6      p' = nr y | c = p y     s = e y          r = r2 y
//
// with p, c1 the sweep's state, e and d the entries the step consumes, ee =
// e^2, a = d - mu, y0 the hardware seed of 1/sqrt(r2) and y its
// third-order correction. p' = gam'/c with gam' = c^2 a - s^2 gam is computed
// as (p a - ee c1)/r, the same number since gam = p c1: it needs no division
// and no case for c = 0. The chase of one matrix of order 64 (4840 rotations)
// took about 8 ms with one lane per matrix, where a rotation was 58 FP64
// slots in a row, and takes 2.0 ms; 750 cycles a rotation, of which the six
// slots are 384 and the rsqrt seed and the two shuffles on the path 230.
constexpr int kGL = 4;          // lanes per matrix
constexpr int kGM = 32 / kGL;   // matrices per warp, at most
// Matrices per warp unless a plan's autotuner chose another count: the groups
// of a warp wait for one another between sweeps, and fewer of them cost more
// FP64 slots in all. 512 matrices of order 128: 7.8, 8.9, 11.3 and 15.9 ms
// for 1, 2, 4 and 8; 4096 of orders 8 .. 128 with everything else that runs
// beside the chase: 42.8, 39.5, 40.9 and 44.3 ms.
constexpr int kGrpDefault = 2;

// Sign flips and selects on the integer halves: a negated or selected FP64
// register otherwise costs an FP64 slot.
GLA_DEV double flip(double x, unsigned mask) {
  return __hiloint2double((int)((unsigned)__double2hiint(x) ^ mask), __double2loint(x));
}
GLA_DEV double pick(bool f, double x, double y) {
  return __hiloint2double(f ? __double2hiint(x) : __double2hiint(y), f ? __double2loint(x) : __double2loint(y));
}
GLA_DEV int hi_exp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// The shift of :271-273 / :324-326, mu = d0 - e / (m + sign(m) hypot(m, 1))
// with m = (d1 - d0) / 2e, as d0 - 2 e^2 / (dd + sign(dd) sqrt(dd^2 + 4 e^2)),
// dd = d1 - d0.
GLA_DEV double wilkinson_shift(double d0, double d1, double e) {
  const double dd = d1 - d0;
  const double ee4 = (2.0 * e) * (2.0 * e);
  const double q = fma(dd, dd, ee4);
  const int be = hi_exp(q);
  if (be < 1023 - 900 || be > 1023 + 900 || hi_exp(ee4) < 1023 - 1000) {
    const double m = div_fast(dd, 2.0 * e);
    return d0 - div_fast(e, m + tcopysign(hypot1_fast(m), m));
  }
  return fma(-0.5 * ee4, rcp64(dd + copysign(sqrt64(q), dd)), d0);
}

constexpr int kGRows = kSmallMaxN + 4;  // rows of d and of e in shared memory: two of padding on either side
constexpr int kGFlags = kSmallMaxN + 8;  // bytes of deflation flags per matrix, two of padding before
size_t chase_grp_smem_bytes() { return (size_t)kGM * ((2 * kGRows + 3) * sizeof(double) + kGFlags); }

template <int ALGO>
__global__ void __launch_bounds__(32) k_chase_grp(const SmallDesc* __restrict__ descs, const int* __restrict__ perm,
                                                  int count, double* __restrict__ dg_all, double* __restrict__ eg_all,
                                                  ChaseState* __restrict__ cst, double* __restrict__ rot,
                                                  unsigned* __restrict__ hdr, int* __restrict__ info, double tol,
                                                  int max_sweeps_per_n, int* __restrict__ pending,
                                                  unsigned long long* __restrict__ stats, int mats_per_warp) {
  constexpr bool QL = ALGO == kAlgoQL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x, grp = lane / kGL, role = lane % kGL, g0 = grp * kGL;
  const int slot = blockIdx.x * mats_per_warp + grp;
  const bool have = grp < mats_per_warp && slot < count;
  const int mid = have ? perm[slot] : 0;
  SmallDesc dsc;
  dsc.n = 0;
  if (have) dsc = descs[mid];
  const int n = dsc.n;
  int nmax = n;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nmax = max(nmax, __shfl_xor_sync(kAll, nmax, o));
  // d, e of the group's matrix (rows of kGM matrices), and one byte per
  // entry of e: negligible (1), not (0), or to be tested exactly (2)
  double* D = reinterpret_cast<double*>(smem_raw) + 2 * kGM + grp;
  double* E = D + (size_t)kGRows * kGM;
  unsigned char* F = smem_raw + (size_t)(2 * kGRows + 3) * kGM * sizeof(double) + grp * kGFlags + 2;
#define DD(i) D[(size_t)(i) * kGM]
#define EE(i) E[(size_t)(i) * kGM]
  ChaseState st;
  st.status = kChaseDone;
  st.nsweeps = st.bs = 0;
  if (have) st = cst[mid];
  const bool was_running = have && st.status == kChaseRunning;
  bool active = was_running;
  double* dg = dg_all + dsc.w_off;
  double* eg = eg_all + dsc.w_off;
  const int tol_e = prec<double>::biased_exp(tol) - prec<double>::expbias;
  if (active)
    for (int k = role; k < n; k += kGL) {
      DD(k) = dg[k];
      EE(k) = eg[k];
    }
  __syncwarp();
  const unsigned gm = 0xfu << g0;
  if (active)
    for (int j = role; j + 1 < n; j += kGL) F[j] = (unsigned char)negligible_fast(EE(j), DD(j), DD(j + 1), tol_e);
  __syncwarp();
  // The first j >= from with e[j] negligible, else n - 1 (the group together,
  // four entries at a time; undecided ones are tested on the values as they
  // stand, the ones the last sweep left).
  auto first_nf = [&](int from) -> int {
    for (int j0 = from; j0 < n - 1; j0 += kGL) {
      const int j = j0 + role;
      bool f = false;
      if (j < n - 1) {
        const int v = F[j];
        f = v == 1 || (v == 2 && negligible(EE(j), DD(j), DD(j + 1), tol, tol_e));
      }
      const unsigned m = (__ballot_sync(gm, f) >> g0) & 0xfu;
      if (m) return j0 + __ffs(m) - 1;
    }
    return n - 1;
  };
  const int cap = max_sweeps_per_n * n;
  int bs = st.bs, nsw = st.nsweeps, nrot = 0, nhdr = 0;
  double* myrot = rot + 2 * dsc.rot_off;
  unsigned* myhdr = hdr + dsc.hdr_off;
  bool insweep = false, stopped_full = false;
  bool wild = false;  // the sweep meets values outside the fast rotation's range
  int i = 0, be = 0, left = 0;  // left: steps of the sweep still to do
  double mu = 0, p = 0, c = 1, s = 0, sp = 0, r = 0;
  double ei = 0, ee = 0, a = 0, di = 0, t = 0, d_up = 0, e_end = 0;
  int pend = -1;  // row whose d (and e) the last step left to the next one's lane 3
  int iters = 0;
  const int iter_cap = (max_sweeps_per_n + 4) * 4 * nmax * nmax + 64;  // hard bound on loop trips
  while (__any_sync(kAll, active)) {
    if (++iters > iter_cap) {  // defensive: never reached when the sweep cap works
      if (active) {
        if (role == 0) info[mid] = max(1, n - 1);
        active = false;
        st.status = kChaseDone;
      }
      continue;
    }
    if (active && !insweep) {
      if (bs >= n - 1) {
        active = false;
        st.status = kChaseDone;
      } else {
        be = first_nf(bs);
        if (bs == be) {
          bs += 1;
        } else if (bs + 1 == be) {
          if (nrot + 1 > dsc.rot_cap || nhdr + 1 > dsc.hdr_cap) {
            active = false;
            stopped_full = true;
          } else {
            // eig2x2! (:136-161)
            const double dj = DD(bs), dj1 = DD(be), ej = EE(bs);
            const double r1 = (dj + dj1) / 2;
            const double r2 = hypot_borges(dj - dj1, 2 * ej) / 2;
            const double lp = r1 + r2, lm = r1 - r2;
            double cc, ss;
            if (is_zero(ej)) {
              cc = 1;
              ss = 0;
            } else if (tabs(lp - dj) > tabs(lm - dj)) {
              cc = prec<double>::div_ieee(-ej, hypot_borges(ej, lp - dj));
              ss = prec<double>::sqrt_ieee(1 - cc * cc);
            } else {
              ss = prec<double>::div_ieee(tabs(ej), hypot_borges(ej, lm - dj));
              cc = tcopysign(prec<double>::sqrt_ieee(1 - ss * ss), -ej);
            }
            __syncwarp(gm);
            if (role == 0) {
              DD(bs) = lp;
              DD(be) = lm;
              EE(bs) = 0;
              myhdr[nhdr] = pack_hdr(bs, 1, 0);
              myrot[2 * nrot] = cc;
              myrot[2 * nrot + 1] = ss;
            }
            if (role == 0) {
              F[bs] = 1;
              if (be <= n - 2) F[be] = (unsigned char)negligible_fast(EE(be), lm, DD(be + 1), tol_e);
            }
            nhdr++;
            nrot++;
            bs += 2;
          }
        } else if (nsw >= cap) {
          if (role == 0) {
            int cnt = 0;
            for (int b = 0; b + 1 < n; b++) cnt += !negligible(EE(b), DD(b), DD(b + 1), tol, tol_e);
            info[mid] = max(cnt, 1);
          }
          active = false;
          st.status = kChaseDone;
        } else if (nrot + (be - bs) > dsc.rot_cap || nhdr + 1 > dsc.hdr_cap) {
          active = false;
          stopped_full = true;
        } else {
          // shift (:271-273 QL, :324-326 QR) and the start of a chase
          if (QL) {
            mu = wilkinson_shift(DD(bs), DD(bs + 1), EE(bs));
            p = DD(be) - mu;
            i = be - 1;
            ei = EE(i);
            di = DD(i);
            d_up = be + 1 <= n - 1 ? DD(be + 1) : 0.0;
            e_end = be <= n - 2 ? EE(be) : 0.0;
            if (role == 0) myhdr[nhdr] = pack_hdr(be - 1, be - bs, 0);
          } else {
            mu = wilkinson_shift(DD(be), DD(be - 1), EE(be - 1));
            p = DD(bs) - mu;
            i = bs + 1;
            ei = EE(bs);
            di = DD(i);
            d_up = DD(bs);
            e_end = EE(bs - 1);  // (row -1: padding)
            if (role == 0) myhdr[nhdr] = pack_hdr(bs + 1, be - bs, 1);
          }
          nhdr++;
          ee = ei * ei;
          a = di - mu;
          c = 1;
          s = 0;
          left = be - bs;
          pend = -1;
          {  // 2^-480 <= |e| and everything below 2^400: r^2 = p^2 + e^2 and p a stay normal
            bool w = false;
            for (int k = bs + role; k <= be; k += kGL) {
              const int xe = hi_exp(EE(k)), xd = hi_exp(DD(k));
              w |= xd > 1023 + 400 || (k < be && (xe < 1023 - 480 || xe > 1023 + 400));
            }
            wild = __any_sync(gm, w || hi_exp(mu) > 1023 + 400);
          }
          insweep = true;
          nsw++;
        }
      }
    }
    __syncwarp();
    // sweep steps without a vote: as many as every active group still has
    // (groups without a matrix step along on values that nobody reads)
    int steps = 0;
    if (__all_sync(kAll, !active || insweep)) steps = __reduce_min_sync(kAll, active ? left : 0x7fffffff);
    if (steps == 0x7fffffff) steps = 0;
    iters += steps;
    const bool l0 = role == 0, l01 = role < 2, l2 = role == 2, l3 = role == 3;
    const bool any_wild = __any_sync(kAll, active && wild);
    const int adv = active ? (QL ? -kGM : kGM) : 0;
    const double n_mu = flip(mu, 0x80000000u);
    const double c4 = pick(l0, 0.5, pick(l2, n_mu, 0.0));
    double* rp = myrot + 2 * nrot + (role - 1);  // lanes 1 (c) and 2 (s) write the log
    const bool logs = active && (role == 1 || l2);
    double X1 = pick(l2, ee, p), Y1 = pick(l01, p, c), Z1 = pick(l01, ee, 0.0);
    double* dp = active ? &DD(i) : D;  // the row whose d the step consumes
    constexpr int kNx = QL ? -kGM : kGM;  // to the next row
    // Lane 3 stores what the step before left (its d, its e, the flag of that
    // e) at wp, without a branch: the other lanes, and the first step of a
    // sweep, store at a place that nobody reads. edge: the block's boundary
    // entry of e, which the second step stores back as it was.
    double* const junk = E + (size_t)(kGRows - 2) * kGM - (size_t)kGRows * kGM;
    const bool w3 = active && l3;
    double* wp = w3 && pend >= 0 ? &DD(pend) : junk;
    constexpr int kEw = kGRows * kGM - (QL ? 0 : kGM);  // from the row's d to that e
    const int edge = QL ? be : bs;
    for (int step = 0; step < steps; step++) {
      // the next entries (at the sweep's end: the padding's or the next block's, unused)
      const double d_nx = dp[kNx];
      const double e_nx = dp[(QL ? kNx : 0) + kGRows * kGM];
      // 1
      const double v1 = fma(X1, Y1, Z1);
      // the rotation's sign: -1 when |p| > |e| and p < 0, or p = 0 and e < 0
      const unsigned long long bp = prec<double>::bits(p) << 1, be2 = prec<double>::bits(ei) << 1;
      const unsigned neg = ((unsigned)__double2hiint(p) & (bp > be2 ? 0x80000000u : 0u)) |
                           ((unsigned)__double2hiint(ei) & (bp == 0 ? 0x80000000u : 0u));
      const double y0 = flip(rsqrt_seed64(v1), neg);
      // 2
      const double v2 = fma(pick(l01, v1, pick(l2, p, t)), pick(l01, y0, pick(l2, a, 1.0)),
                            pick(l01, 0.0, flip(v1, 0x80000000u)));
      const double r2 = __shfl_sync(kAll, v1, 0, kGL);
      const double y0b = __shfl_sync(kAll, y0, 0, kGL);
      // 3
      const double v3 = fma(pick(l01, flip(v2, 0x80000000u), pick(l2, e_nx, di)), pick(l01, y0, pick(l2, e_nx, 1.0)),
                            pick(l01, 1.0, pick(l2, 0.0, v1)));
      const double nr = __shfl_sync(kAll, v2, 2, kGL);
      // 4
      const double v4 = fma(pick(l0, v3, pick(role == 1, y0, pick(l2, d_nx, sp))),
                            pick(l0, 0.375, pick(role == 1, v3, pick(l2, 1.0, r))), c4);
      const double ee_nx = __shfl_sync(kAll, v3, 2, kGL);
      const double q = __shfl_sync(kAll, v4, 0, kGL);
      const double ye = __shfl_sync(kAll, v4, 1, kGL);
      const double a_nx = __shfl_sync(kAll, v4, 2, kGL);
      // 5
      const double y = fma(ye, q, y0b);
      // what the last step left: its d (v2) and e (v4) in lane 3
      const double e_set = pick(pend == edge, e_end, v4);
      wp[0] = v2;
      wp[kEw] = e_set;
      F[w3 ? (QL ? pend : pend - 1) : -2] = (unsigned char)negligible_fast(e_set, v2, d_up, tol_e);
      d_up = pick(pend >= 0, v2, d_up);
      // 6
      double v6 = pick(l0, nr, pick(role == 1, p, pick(l2, ei, r2))) * y;
      if (any_wild) {  // r^2 or the products may leave the normal range: the scalar rotation
        if (wild) {
          double cc, ss, rr;
          givens(p, ei, cc, ss, rr);
          const double pn = cc * a - ss * (ei * c);
          v6 = l0 ? pn : (role == 1 ? cc : (l2 ? ss : rr));
        }
        __syncwarp();
      }
      if (logs) *rp = v6;
      rp += 2;
      const double pn = __shfl_sync(kAll, v6, 0, kGL);
      const double Yn = __shfl_sync(kAll, v6, l01 ? 0 : 1, kGL);
      const double sn = __shfl_sync(kAll, v6, 2, kGL);
      t = v3;
      sp = s;
      r = v6;
      pend = QL ? i + 1 : i - 1;
      wp = w3 ? dp - kNx : junk;
      i += QL ? -1 : 1;
      dp += adv;
      p = pn;
      s = sn;
      if (any_wild) c = __shfl_sync(kAll, v6, 1, kGL);
      ei = e_nx;
      di = d_nx;
      a = a_nx;
      X1 = pick(l2, ee_nx, pn);
      Y1 = Yn;
      Z1 = pick(l01, ee_nx, 0.0);
      ee = ee_nx;
    }
    if (steps > 0) {
      c = __shfl_sync(kAll, Y1, 2, kGL);
      if (active) {
        nrot += steps;
        left -= steps;
      }
    }
    if (active && insweep && left == 0) {
      // the sweep's end: gam = p c, e[end] = s p, and what the last step left
      const double w1 = pick(l2, s, pick(l3, sp, p)) * pick(l2, p, pick(l3, r, c));
      const double gam = __shfl_sync(gm, w1, 0, kGL);
      const double eb = __shfl_sync(gm, w1, 2, kGL);
      const double w2 = pick(l3, t, mu) + flip(gam, l3 ? 0x80000000u : 0u);
      const double db = __shfl_sync(gm, w2, 0, kGL);
      if (l3) {
        const bool inner = QL ? pend < be : pend > bs;
        DD(pend) = w2;
        if (QL) {  // pend = bs + 1
          if (inner) EE(pend) = w1;
          EE(bs) = eb;
          DD(bs) = db;
          if (pend <= n - 2) F[pend] = (unsigned char)negligible_fast(inner ? w1 : e_end, w2, d_up, tol_e);
          F[bs] = (unsigned char)negligible_fast(eb, db, w2, tol_e);
        } else {  // pend = be - 1
          if (inner) {
            EE(pend - 1) = w1;
            F[pend - 1] = (unsigned char)negligible_fast(w1, d_up, w2, tol_e);
          }
          EE(be - 1) = eb;
          DD(be) = db;
          F[be - 1] = (unsigned char)negligible_fast(eb, w2, db, tol_e);
          if (be <= n - 2) F[be] = (unsigned char)negligible_fast(EE(be), db, DD(be + 1), tol_e);
        }
      }
      insweep = false;
    }
    __syncwarp();
  }
  __syncwarp();
  if (was_running) {
    for (int k = role; k < n; k += kGL) {
      dg[k] = DD(k);
      eg[k] = EE(k);
    }
    if (role == 0) {
      const int sweeps_this_pass = nsw - st.nsweeps;
      st.bs = bs;
      st.nsweeps = nsw;
      st.nrot = nrot;
      st.nhdr = nhdr;
      cst[mid] = st;
      if (stopped_full) atomicAdd(pending, 1);
      atomicAdd(&stats[0], (unsigned long long)nrot);
      atomicAdd(&stats[1], (unsigned long long)sweeps_this_pass);
      atomicAdd(&stats[2], (unsigned long long)nrot * (unsigned long long)n);
    }
  }
#undef DD
#undef EE
}

template <class T, int ALGO> static void set_chase_attr() {
  cudaFuncSetAttribute(k_chase<T, ALGO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)chase_smem_bytes(kSmallMaxN, (int)sizeof(T)));
}

cudaError_t chase_kernels_init() {
  set_chase_attr<double, kAlgoPWK>();
  set_chase_attr<float, kAlgoQL>();
  set_chase_attr<float, kAlgoQR>();
  set_chase_attr<float, kAlgoPWK>();
  return cudaGetLastError();
}

cudaError_t launch_chase(int tcode, int algo, int count, size_t smem, cudaStream_t st, const SmallDesc* descs,
                         const int* perm, void* d, void* e, ChaseState* cst, void* rot, unsigned* hdr, int* info,
                         double tol, int max_sweeps_per_n, int* pending, unsigned long long* stats,
                         int lanes_per_warp) {
  if (count <= 0) return cudaSuccess;
  // One matrix per lane: FP32 chases are instruction-latency bound, 8 matrices
  // per warp keep the lanes of a warp in step; the FP64 root-free chase pays
  // ~64 cycles per warp instruction, so the cost of divergence and of idle
  // lanes balance at 16. A plan's autotuner may choose another count (1..32).
  const int lpw = (lanes_per_warp >= 1 && lanes_per_warp <= 32) ? lanes_per_warp : (tcode == kF64 ? 16 : 8);
  const int nb = (count + lpw - 1) / lpw;
#define GLA_CH(T, A)                                                                                             \
  k_chase<T, A><<<nb, 32, smem, st>>>(descs, perm, count, (T*)d, (T*)e, cst, (T*)rot, hdr, info, (T)tol,        \
                                      max_sweeps_per_n, pending, stats, lpw)
  if (tcode == kF64 && algo != kAlgoPWK) {
    const int mpw = lanes_per_warp >= 1 ? std::min(lanes_per_warp, kGM) : kGrpDefault;
    const int nbg = (count + mpw - 1) / mpw;
    auto kern = algo == kAlgoQL ? k_chase_grp<kAlgoQL> : k_chase_grp<kAlgoQR>;
    kern<<<nbg, 32, chase_grp_smem_bytes(), st>>>(descs, perm, count, (double*)d, (double*)e, cst,
                                                            (double*)rot, hdr, info, tol, max_sweeps_per_n, pending,
                                                            stats, mpw);
  } else if (tcode == kF64) {
    GLA_CH(double, kAlgoPWK);
  } else {
    if (algo == kAlgoQL) GLA_CH(float, kAlgoQL);
    else if (algo == kAlgoQR) GLA_CH(float, kAlgoQR);
    else GLA_CH(float, kAlgoPWK);
  }
#undef GLA_CH
  return cudaGetLastError();
}

}  // namespace gla
