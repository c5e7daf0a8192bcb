// dg_kernels_common.cu -- table images, layout permutation, RK combinations
// and the device-side CFL step.
#include <cstring>

#include "dg_device.cuh"
#include "dg_launch.h"

namespace dg {

template <int P>
static void fill_tab(const dg_order_tables &s, Tab<P> *t) {
  constexpr int NP = Tab<P>::NP, NQ = Tab<P>::NQ, N1 = Tab<P>::N1;
  for (int q = 0; q < NQ; q++) {
    for (int i = 0; i < NP; i++) {
      t->B[q][i] = s.B[q][i];
      t->GR[q][i] = s.GR[q][i];
      t->GS[q][i] = s.GS[q][i];
    }
    t->r[q] = s.r[q];
    t->s[q] = s.s[q];
    t->w[q] = s.w[q];
  }
  for (int f = 0; f < 3; f++)
    for (int j = 0; j < N1; j++)
      for (int i = 0; i < NP; i++) t->E[f][j][i] = s.E[f][j][i];
  for (int j = 0; j < N1; j++) {
    t->t1[j] = s.t1[j];
    t->w1[j] = s.w1[j];
  }
  for (int v = 0; v < 3; v++)
    for (int i = 0; i < NP; i++) t->V[v][i] = s.V[v][i];
}

size_t tab_bytes(int p) {
  switch (p) {
    case 0: return sizeof(Tab<0>);
    case 1: return sizeof(Tab<1>);
    case 2: return sizeof(Tab<2>);
    case 3: return sizeof(Tab<3>);
    case 4: return sizeof(Tab<4>);
    case 5: return sizeof(Tab<5>);
  }
  return 0;
}

void build_tab(int p, const dg_order_tables &src, void *dst) {
  switch (p) {
    case 0: fill_tab<0>(src, static_cast<Tab<0> *>(dst)); break;
    case 1: fill_tab<1>(src, static_cast<Tab<1> *>(dst)); break;
    case 2: fill_tab<2>(src, static_cast<Tab<2> *>(dst)); break;
    case 3: fill_tab<3>(src, static_cast<Tab<3> *>(dst)); break;
    case 4: fill_tab<4>(src, static_cast<Tab<4> *>(dst)); break;
    case 5: fill_tab<5>(src, static_cast<Tab<5> *>(dst)); break;
  }
}

static constexpr int kB = 256;
static unsigned grid_for(size_t n) { return (unsigned)((n + kB - 1) / kB); }

// Layout permutations: a thread takes one element through kRows rows of the
// state, so its index is read once, kRows loads are in flight, and no index is
// divided (state in / out at 2.1M triangles, p = 3, 40 rows: 380 / 303 us with one
// thread per value and a 64-bit division, 209 / 207 us)
constexpr int kRows = 8;
static dim3 row_grid(int n, int rows) {
  return dim3((unsigned)((n + kB - 1) / kB), (unsigned)((rows + kRows - 1) / kRows));
}

// CMP: also set *changed when any value differs (bitwise) from the one it
// overwrites
template <bool CMP>
__global__ void k_permute_in(const double *__restrict__ user, double *__restrict__ in,
                             const int *__restrict__ perm, int rows, int K, int Kp,
                             int *changed) {
  const int e = blockIdx.x * kB + threadIdx.x;
  if (e >= Kp) return;
  const int r0 = blockIdx.y * kRows, o = e < K ? perm[e] : 0;
  double v[kRows];
#pragma unroll
  for (int r = 0; r < kRows; r++)
    v[r] = e < K && r0 + r < rows ? user[(size_t)(r0 + r) * K + o] : 0.0;
  bool diff = false;
#pragma unroll
  for (int r = 0; r < kRows; r++)
    if (r0 + r < rows) {
      double *p = in + (size_t)(r0 + r) * Kp + e;
      if (CMP) diff |= __double_as_longlong(*p) != __double_as_longlong(v[r]);
      *p = v[r];
    }
  if (CMP && diff) *changed = 1;
}

__global__ void k_permute_out(const double *__restrict__ in, double *__restrict__ user,
                              const int *__restrict__ perm, int rows, int K, int Kp) {
  const int e = blockIdx.x * kB + threadIdx.x;
  if (e >= K) return;
  const int r0 = blockIdx.y * kRows, o = perm[e];
  double v[kRows];
#pragma unroll
  for (int r = 0; r < kRows; r++) v[r] = r0 + r < rows ? in[(size_t)(r0 + r) * Kp + e] : 0.0;
#pragma unroll
  for (int r = 0; r < kRows; r++)
    if (r0 + r < rows) user[(size_t)(r0 + r) * K + o] = v[r];
}

void launch_permute_in(cudaStream_t st, const double *user, double *internal, const int *perm,
                       int rows, int K, int Kp) {
  if (rows > 0 && Kp > 0)
    k_permute_in<false><<<row_grid(Kp, rows), kB, 0, st>>>(user, internal, perm, rows, K, Kp,
                                                           nullptr);
}

void launch_permute_in_cmp(cudaStream_t st, const double *user, double *internal,
                           const int *perm, int rows, int K, int Kp, int *changed) {
  if (rows > 0 && Kp > 0)
    k_permute_in<true><<<row_grid(Kp, rows), kB, 0, st>>>(user, internal, perm, rows, K, Kp,
                                                          changed);
}

void launch_permute_out(cudaStream_t st, const double *internal, double *user, const int *perm,
                        int rows, int K, int Kp) {
  if (rows > 0 && K > 0)
    k_permute_out<<<row_grid(K, rows), kB, 0, st>>>(internal, user, perm, rows, K, Kp);
}

__global__ void k_xpay(int n, const double *x, double a, const double *y, double *z) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) z[i] = x[i] + a * y[i];  // rk_tempstorage, time_integrator.cu:107-113
}
__global__ void k_rk4_final(int n, double *c, const double *__restrict__ k1,
                            const double *__restrict__ k2, const double *__restrict__ k3,
                            const double *__restrict__ k4) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;  // rk4, time_integrator.cu:124-130
  if (i < n) c[i] += k1[i] / 6. + k2[i] / 3. + k3[i] / 3. + k4[i] / 6.;
}

void launch_xpay(cudaStream_t st, int n, const double *x, double a, const double *y, double *z) {
  if (n) k_xpay<<<grid_for(n), kB, 0, st>>>(n, x, a, y, z);
}
void launch_rk4_final(cudaStream_t st, int n, double *c, const double *k1, const double *k2,
                      const double *k3, const double *k4) {
  if (n) k_rk4_final<<<grid_for(n), kB, 0, st>>>(n, c, k1, k2, k3, k4);
}

__global__ void k_advance_t(DevScalars *ds) { advance_time(ds); }

__global__ void k_batch_put_scalars(BatchProb *pr, const DevScalars *h, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) *pr[i].ds = h[i];
}
__global__ void k_batch_get_scalars(BatchProb *pr, DevScalars *h, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) h[i] = *pr[i].ds;
}
void launch_batch_put_scalars(cudaStream_t st, BatchProb *probs, const DevScalars *h, int n) {
  if (n) k_batch_put_scalars<<<grid_for(n), kB, 0, st>>>(probs, h, n);
}
void launch_batch_get_scalars(cudaStream_t st, BatchProb *probs, DevScalars *h, int n) {
  if (n) k_batch_get_scalars<<<grid_for(n), kB, 0, st>>>(probs, h, n);
}

struct BatchTabsImage {
  Tab<1> t1;
  Tab<2> t2;
  Tab<3> t3;
};
size_t batch_tabs_bytes() { return sizeof(BatchTabsImage); }
void build_batch_tabs(const void *t1, const void *t2, const void *t3, void *dst) {
  BatchTabsImage *b = static_cast<BatchTabsImage *>(dst);
  if (t1) std::memcpy(&b->t1, t1, sizeof(Tab<1>));
  if (t2) std::memcpy(&b->t2, t2, sizeof(Tab<2>));
  if (t3) std::memcpy(&b->t3, t3, sizeof(Tab<3>));
}

void launch_advance_t(cudaStream_t st, DevScalars *ds) { k_advance_t<<<1, 1, 0, st>>>(ds); }

}  // namespace dg
