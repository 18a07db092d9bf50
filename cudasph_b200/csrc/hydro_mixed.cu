// hydro_mixed.cu -- the mixed-precision form of the density and hydro loops.
//
// Neighbour records are gathered as in the FP64 form; the pair separation
// and velocity difference are formed in FP64 (exact differences of the FP64
// coordinates, rounded once), and everything that varies per pair -- the
// distance, u, the kernel functions, the artificial viscosity and the pair
// vectors -- runs in FP32 with compensated (Kahan-Babuska) float sums.  The
// factors that are constant over a particle's pairs (1/h^5, 1/h^2, P/rho^2,
// the grad-h terms, m_i) are applied in FP64 to those sums, and u = r (2 /
// range) takes the per-particle scale as a float-float pair: rounding such a
// constant to FP32 would bias every pair of that particle the same way, and
// in near-hydrostatic stars, where the pair forces largely cancel, such a
// bias (unlike the random per-pair rounding) grows into the net force.  The
// j-side pair force is assembled in FP64 from the FP32 pair vectors and the
// owner's FP64 factors; outputs and atomics stay FP64.
#include "common.cuh"
#include "sphpair.cuh"

namespace sph {


struct KSum {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float s = hi + v;
    const float bp = s - hi;
    lo += (hi - (s - bp)) + (v - bp);
    hi = s;
  }
  __device__ __forceinline__ double get() const { return (double)hi + (double)lo; }
};

// sum over the S lanes of a particle, in FP64
template <int S>
__device__ __forceinline__ double lanes_sum(const KSum &k) { return sub_sum<S>(k.get()); }

// Lanes per particle, as in the FP64 loops: a list is a row of its own, and
// one lane per particle reads 32 rows at a time (65,536 particles, hydro, us:
// 217, and 164 when the lists of 32 particles were interleaved).  us, density
// / hydro, with 16, 8, 4, 2 lanes and 1: 2,000 particles 12.6 / 18.9 (16), 16.8
// / 23.2 (8), 67 / 101 (1); 16,384 with 8 / 4 / 2 / 1 lanes 31 / 50, 29 / 47,
// 42 / 65, 71 / 109; 65,536 76 / 132, 76 / 127, 89 / 162, 92 / 217; 1,000,000
// 1008 / 1827, 904 / 1661, 867 / 1728, 928 / 2115.
constexpr int kSubSmall = 16, kSmallSet = 8192, kSub = 4;

// x (hi + lo) for a float-float constant: the product to about 2^-46
__device__ __forceinline__ float mul_ff(float x, float hi, float lo) { return fmaf(x, hi, x * lo); }

__device__ __forceinline__ void split_ff(double v, float &hi, float &lo) {
  hi = (float)v;
  lo = (float)(v - (double)hi);
}

template <int S>
__global__ void __launch_bounds__(128) k_density_mixed(HydroArgs a) {
  grid_enter();
  const int s = a.leaf0 * kLeaf + (int)((blockIdx.x * blockDim.x + threadIdx.x) / S), sub = (int)threadIdx.x % S;
  const bool valid = s < min(a.leaf1 * kLeaf, a.n);
  double4 pi = make_double4(0, 0, 0, 0), vi = make_double4(0, 0, 0, 0);
  int cnt = 0;
  if (valid) {
    pi = a.pos[s];
    vi = a.vel[s];
    cnt = min(a.n_ngb[s], a.cap);
  }
  const int *lst = a.list + (size_t)s * a.stride;
  const double w = pi.w;
  float iw_hi = 0.f, iw_lo = 0.f;  // 2 / range as a float-float pair
  if (w > 0) split_ff(2.0 / w, iw_hi, iw_lo);
  KSum dens, om, ps, sdig, div, cx, cy, cz;
  int jn = sub + S < cnt ? ldg(lst + sub + S) : 0;
  double4 pn = make_double4(0, 0, 0, 0), vn = pn;
  if (sub < cnt) {
    const int j0 = ldg(lst + sub);
    pn = ld4(a.pos + j0);
    vn = ld4(a.vel + j0);
  }
  for (int k = sub; k < cnt; k += S) {
    {
      const double4 pj = pn, vj = vn;
      if (k + S < cnt) {
        pn = ld4(a.pos + jn);
        vn = ld4(a.vel + jn);
        if (k + 2 * S < cnt) jn = ldg(lst + k + 2 * S);
      }
      const float dx = (float)(pi.x - pj.x), dy = (float)(pi.y - pj.y), dz = (float)(pi.z - pj.z);
      const float u = mul_ff(sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx))), iw_hi, iw_lo);
      const float mj = (float)vj.w;
      dens.add(mj * k_w<float>(u));
      om.add(mj * k_dwdh<float>(u));
      ps.add(mj * k_dphidh<float>(u));
      sdig.add(-k_digdh<float>(u));
      const float dvx = (float)(vi.x - vj.x), dvy = (float)(vi.y - vj.y), dvz = (float)(vi.z - vj.z);
      const float wt = mj * k_dw<float>(u);
      div.add(wt * (dx * dvx + dy * dvy + dz * dvz));
      cx.add(wt * (dy * dvz - dz * dvy));
      cy.add(wt * (dz * dvx - dx * dvz));
      cz.add(wt * (dx * dvy - dy * dvx));
    }
  }
  __syncwarp();
  double de = lanes_sum<S>(dens), o = lanes_sum<S>(om), p = lanes_sum<S>(ps), dv = lanes_sum<S>(div);
  const double sd = lanes_sum<S>(sdig), X = lanes_sum<S>(cx), Y = lanes_sum<S>(cy), Z = lanes_sum<S>(cz);
  if (!valid || sub != 0) return;
  if (a.dsum) a.dsum[s] = make_double4(sd, X, Y, Z);
  double4 d = make_double4(0, 0, 0, 0);
  double rho = 0;
  if (w > 0 && cnt > 0) {
    const double h = 0.5 * w;
    const double h3 = h * h * h, h5 = h3 * h * h;
    if (sd != 0) {
      o *= 1.0 / h3 / sd;
      p *= 1.0 / h / sd;
    } else {
      o = p = 0;
    }
    de *= 1.0 / h3;
    dv = dv / de / h5;
    const double c = sqrt(X * X + Y * Y + Z * Z) / de / h5;
    rho = de;
    d = make_double4(dv, c, o, p);
  }
  a.hyd[s].x = rho;
  a.dd[s] = d;
}

// Hydro (dev_hydro_dots.cu:25-113 with dev_art_visc.cu:8-32): with
// A = P_i / rho_i^2 the i-side force is
//   a_i = -[A S1 + S2 / 2] / h^5 + K [S3] / h^2,  K = A omega_i + psi_i / 2,
//   S1 = sum_j m_j dw(u) r_ij,  S2 = sum_j m_j Pi_ij dw(u) r_ij,
//   S3 = sum_j dig(u) r_ij,
// du_i/dt = [A T1 + T2 / 2] / h^5 - A omega_i T3 / h^2 with the same sums of
// r_ij . v_ij in place of r_ij; the pair's force on j, m_i acc_ij (r_i - r_j),
// is assembled in FP64 from the FP32 pair vectors dw r_ij, Pi dw r_ij, dig r_ij.
template <int S>
__global__ void __launch_bounds__(128) k_hydro_mixed(HydroArgs a) {
  grid_enter();
  const int s = a.leaf0 * kLeaf + (int)((blockIdx.x * blockDim.x + threadIdx.x) / S), sub = (int)threadIdx.x % S;
  const bool valid = s < min(a.leaf1 * kLeaf, a.n);
  double4 pi = make_double4(0, 0, 0, 0), vi = make_double4(0, 0, 0, 1), hi4 = make_double4(0, 0, 0, 0),
          di = make_double4(0, 0, 0, 0), fi = make_double4(0, 0, 0, 0);
  int cnt = 0;
  if (valid) {
    pi = a.pos[s];
    vi = a.vel[s];
    hi4 = a.hyd[s];
    di = a.dd[s];
    fi = a.aux[s];
    cnt = min(a.n_ngb[s], a.cap);
  }
  const int *lst = a.list + (size_t)s * a.stride;
  const double hh = 0.5 * pi.w;
  float ih_hi = 0.f, ih_lo = 0.f;  // 1 / h as a float-float pair
  if (hh > 0) split_ff(1.0 / hh, ih_hi, ih_lo);
  const double prho2 = (hi4.x > 0) ? hi4.y / (hi4.x * hi4.x) : 0;
  const double h2 = hh * hh, h5 = h2 * h2 * hh;
  const double ih5 = hh > 0 ? 1.0 / h5 : 0.0, ih2 = hh > 0 ? 1.0 / h2 : 0.0;
  const double psi_i = a.use_psi ? di.w : 0;
  const double K = prho2 * di.z + 0.5 * psi_i;
  // the owner's factors of the j-side force m_i acc_ij (FP64)
  const double mi = vi.w;
  const double c1 = mi * prho2 * ih5, c2 = 0.5 * mi * ih5, c3 = mi * K * ih2;
  const float alpha = (float)a.alpha, beta = (float)a.beta;
  const float ci = (float)fi.x, pr_i = (float)fi.y, bal_i = (float)fi.z;
  KSum s1x, s1y, s1z, s2x, s2y, s2z, s3x, s3y, s3z, t1, t2, t3;
  float vmax = 0.f;
  for (int k = sub; k < cnt; k += S) {
    {
      const int j = ldg(lst + k);
      const double4 pj = ld4(a.pos + j), vj = ld4(a.vel + j), fj = ld4(a.aux + j);
      const float dx = (float)(pi.x - pj.x), dy = (float)(pi.y - pj.y), dz = (float)(pi.z - pj.z);
      const float dvx = (float)(vi.x - vj.x), dvy = (float)(vi.y - vj.y), dvz = (float)(vi.z - vj.z);
      const float ds = sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
      const float u = mul_ff(ds, ih_hi, ih_lo);
      const float drdv = fmaf(dz, dvz, fmaf(dy, dvy, dx * dvx));
      // artificial viscosity on the per-particle factors {c, P / rho^2, B}
      const float cj = (float)fj.x;
      float visc = 0.f, vs = ci + cj;
      if (drdv < 0.f) {
        const float mu0 = drdv / ds;
        vs -= beta * mu0;
        const float mu = mu0 / (ci + cj) * (bal_i + (float)fj.z);
        visc = (pr_i + (float)fj.y) * (-alpha * mu + beta * mu * mu);
      }
      vmax = fmaxf(vmax, vs);
      const float dwu = k_dw<float>(u), digu = k_dig<float>(u);
      const float mj = (float)vj.w;
      const float mdw = mj * dwu, mpdw = visc * mdw;
      const float e1x = mdw * dx, e1y = mdw * dy, e1z = mdw * dz;     // m_j dw r_ij
      const float e2x = mpdw * dx, e2y = mpdw * dy, e2z = mpdw * dz;  // m_j Pi dw r_ij
      const float e3x = digu * dx, e3y = digu * dy, e3z = digu * dz;  // dig r_ij
      s1x.add(e1x); s1y.add(e1y); s1z.add(e1z);
      s2x.add(e2x); s2y.add(e2y); s2z.add(e2z);
      s3x.add(e3x); s3y.add(e3y); s3z.add(e3z);
      t1.add(mdw * drdv);
      t2.add(mpdw * drdv);
      t3.add(digu * drdv);
      if (a.jside && j != s) {
        // m_i acc_ij r_ij = [c1 m_j dw r + c2 m_j Pi dw r] / m_j - c3 dig r / m_j
        const double imj = fj.w;
        const double f1 = c1 * imj, f2 = c2 * imj, f3 = c3 * imj;
        atomicAdd(&a.dots[j].x, f1 * e1x + f2 * e2x - f3 * e3x);
        atomicAdd(&a.dots[j].y, f1 * e1y + f2 * e2y - f3 * e3y);
        atomicAdd(&a.dots[j].z, f1 * e1z + f2 * e2z - f3 * e3z);
      }
    }
  }
  __syncwarp();
  const double ax = -(prho2 * lanes_sum<S>(s1x) + 0.5 * lanes_sum<S>(s2x)) * ih5 + K * ih2 * lanes_sum<S>(s3x);
  const double ay = -(prho2 * lanes_sum<S>(s1y) + 0.5 * lanes_sum<S>(s2y)) * ih5 + K * ih2 * lanes_sum<S>(s3y);
  const double az = -(prho2 * lanes_sum<S>(s1z) + 0.5 * lanes_sum<S>(s2z)) * ih5 + K * ih2 * lanes_sum<S>(s3z);
  const double du = (prho2 * lanes_sum<S>(t1) + 0.5 * lanes_sum<S>(t2)) * ih5 - prho2 * di.z * ih2 * lanes_sum<S>(t3);
  const double vs = sub_max<S>((double)vmax);
  if (!valid || sub != 0) return;
  atomicAdd(&a.dots[s].x, ax);
  atomicAdd(&a.dots[s].y, ay);
  atomicAdd(&a.dots[s].z, az);
  a.dots[s].w = du;
  a.vsig[s] = vs;
}

int launch_density_mixed(const HydroArgs &a, cudaStream_t st) {
  if (a.leaf1 <= a.leaf0) return 0;
  const int n = (a.leaf1 - a.leaf0) * kLeaf;
  if (n < kSmallSet) launch(k_density_mixed<kSubSmall>, (n * kSubSmall + 127) / 128, 128, st, a);
  else launch(k_density_mixed<kSub>, (n * kSub + 127) / 128, 128, st, a);
  return 1;
}
int launch_hydro_prep(int n, const double4 *pos, const double4 *vel, const double4 *hyd, const double4 *dd,
                      double gamma, double4 *aux, double4 *dots, cudaStream_t st);

int launch_hydro_mixed(const HydroArgs &a, cudaStream_t st) {
  // every particle's factors {c, P / rho^2, B, 1 / m}: a shard's pairs reach outside its own leaves, and
  // a shard without leaves still clears the sums that the shards add up
  int launches = launch_hydro_prep(a.n, a.pos, a.vel, a.hyd, a.dd, a.gamma, a.aux, a.dots, st);
  if (a.leaf1 <= a.leaf0) return launches;
  const int n = (a.leaf1 - a.leaf0) * kLeaf;
  if (n < kSmallSet) launch(k_hydro_mixed<kSubSmall>, (n * kSubSmall + 127) / 128, 128, st, a);
  else launch(k_hydro_mixed<kSub>, (n * kSub + 127) / 128, 128, st, a);
  return launches + 1;
}

}  // namespace sph
