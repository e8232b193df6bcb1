// Size-field producers on the device: element gradients of vertex fields
// (element_gradients.cpp:15-91 with jacobian.cpp:7-66), recovery of element
// fields to vertices weighted by element volume (recover_by_volume.cpp:10-68),
// an isotropic size from recovered Hessians (size_from_hessian.cpp:12-72), and
// warping coordinates as far as a quality floor allows
// (warp_to_limit.cpp:14-81). Every arithmetic step follows the reference's
// order, so results are bit-identical to its CPU build.
#include <cfloat>
#include <string>

#include "fields.hpp"

namespace osh {

namespace {

// algebra.hpp's helpers, in their operation order
__device__ inline void cross_ref(double const* a, double const* b, double* c)
{
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ inline double dot_ref(double const* a, double const* b, u32 n)
{
  double d = 0;
  for (u32 i = 0; i < n; ++i) d += a[i] * b[i];
  return d;
}

// invert_jacobian (jacobian.cpp:20-61) for 1-, 2- and 3-simplices
__device__ void invert_jacobian(u32 dim, double in[3][3], double out[3][3])
{
  if (dim == 3) {
    // invert_3x3 (algebra.hpp): cofactor rows scaled by 1/det, transposed
    double tmp[3][3], c[3];
    cross_ref(in[0], in[1], c);
    double d = dot_ref(in[2], c, 3);
    cross_ref(in[1], in[2], tmp[0]);
    cross_ref(in[2], in[0], tmp[1]);
    cross_ref(in[0], in[1], tmp[2]);
    double s = 1.0 / d;
    for (u32 i = 0; i < 3; ++i)
      for (u32 j = 0; j < 3; ++j) tmp[i][j] = tmp[i][j] * s;
    for (u32 i = 0; i < 3; ++i)
      for (u32 j = 0; j < 3; ++j) out[i][j] = tmp[j][i];
  } else if (dim == 2) {
    double nrm[2][2];
    for (u32 i = 0; i < 2; ++i)
      for (u32 j = 0; j < 2; ++j) {
        nrm[i][j] = 0;
        for (u32 k = 0; k < 3; ++k) nrm[i][j] += in[i][k] * in[j][k];
      }
    double d = nrm[0][0] * nrm[1][1] - nrm[0][1] * nrm[1][0];
    double inv[2][2] = {{nrm[1][1] / d, -nrm[0][1] / d}, {-nrm[1][0] / d, nrm[0][0] / d}};
    for (u32 i = 0; i < 3; ++i)
      for (u32 j = 0; j < 3; ++j) out[i][j] = 0;
    for (u32 i = 0; i < 3; ++i)
      for (u32 j = 0; j < 2; ++j)
        for (u32 k = 0; k < 2; ++k) out[i][j] += in[k][i] * inv[k][j];
  } else {
    double msq = dot_ref(in[0], in[0], 3);
    for (u32 i = 0; i < 3; ++i) out[i][0] = in[0][i] / msq;
    for (u32 i = 0; i < 3; ++i)
      for (u32 j = 1; j < 3; ++j) out[i][j] = 0;
  }
}

// Gradients of one element's fields: the inverse Jacobian and, per component,
// the sum over the edges from vertex 0 in their order (element_gradients.cpp).
// NC: the components at compile time (0: nc of them), so that a gradient is
// summed in registers; `put` takes value k of the element's nc * 3.
template <u32 NC, class Put>
__device__ inline void element_gradient(u32 dim, u32 const* ve, double const* __restrict__ x,
    u32 nc_any, double const* __restrict__ f, Put put)
{
  u32 const vpe = dim + 1, nc = NC ? NC : nc_any;
  double ex[4][3];
#pragma unroll
  for (u32 j = 0; j < 4; ++j)
    if (j < vpe) load3(x, ve[j], ex[j]);
  // element_jacobian: column j is x[j+1] - x[0]
  double jac[3][3];
#pragma unroll
  for (u32 a = 0; a < 3; ++a)
#pragma unroll
    for (u32 b = 0; b < 3; ++b) jac[b][a] = a < dim ? ex[a + 1][b] - ex[0][b] : 0;
  double jaci[3][3];
  invert_jacobian(dim, jac, jaci);
#pragma unroll
  for (u32 k = 0; k < (NC ? NC : nc); ++k) {
    double fv[4];
#pragma unroll
    for (u32 j = 0; j < 4; ++j) fv[j] = j < vpe ? f[(size_t)ve[j] * nc + k] : 0;
#pragma unroll
    for (u32 l = 0; l < 3; ++l) {
      double g = 0;
#pragma unroll
      for (u32 j = 0; j < 3; ++j)
        if (j < dim) g += jaci[j][l] * (fv[j + 1] - fv[0]);
      put(k * 3 + l, g);
    }
  }
}

// A thread per element. Bound by the write of the gradients (24 nc bytes an
// element) once they are written a block at a time through shared memory:
// a thread writing its own element's values put 32 lanes 24 nc bytes apart
// in every store, and the running sums were kept in the output array, read
// and written again for each edge (1.57M tets: nc = 1 and 3 took 418 us
// together, now 79 us, 33 us of it the bytes at copy rate).
constexpr u32 GRAD_BLOCK = 128;

template <u32 DIM, u32 NC>
__global__ void __launch_bounds__(GRAD_BLOCK) k_element_gradients(u32 ne,
    u32 const* __restrict__ voe, double const* __restrict__ x, double const* __restrict__ f,
    double* __restrict__ out)
{
  pdl_wait();
  __shared__ double s_out[GRAD_BLOCK * NC * 3];
  u32 const first = blockIdx.x * GRAD_BLOCK, i = first + threadIdx.x;
  if (i < ne) {
    u32 ve[DIM + 1];
#pragma unroll
    for (u32 j = 0; j <= DIM; ++j) ve[j] = voe[(size_t)i * (DIM + 1) + j];
    double* mine = s_out + threadIdx.x * (NC * 3);  // (an odd stride: no bank conflicts)
    element_gradient<NC>(DIM, ve, x, NC, f, [&](u32 k, double g) { mine[k] = g; });
  }
  __syncthreads();
  u32 const n = (ne - first < GRAD_BLOCK ? ne - first : GRAD_BLOCK) * NC * 3;
  double* o = out + (size_t)first * (NC * 3);
  for (u32 k = threadIdx.x; k < n; k += GRAD_BLOCK) o[k] = s_out[k];
}

// any number of components and dimensions 1 to 3
__global__ void k_element_gradients_any(u32 dim, u32 ne, u32 const* __restrict__ voe,
    double const* __restrict__ x, u32 nc, double const* __restrict__ f,
    double* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ne) return;
  double* g = out + (size_t)i * nc * 3;
  element_gradient<0>(dim, voe + (size_t)i * (dim + 1), x, nc, f,
      [&](u32 k, double v) { g[k] = v; });
}

// A thread per vertex and component: the nc lanes of a vertex read an
// element's nc values side by side (and its size and id from one address),
// and each component is summed over the row in its order, as the reference
// sums it. RECOVER_BATCH elements' loads are issued before any is used:
// the gathers' latency bounds the kernel, the sums are short. (A thread per
// vertex kept its nc sums in the output array, with 32 rows' gathers in
// every load: 1.57M tets, nc = 3 and 9 took 771 us together, now
// 119 us, 38 us of it the bytes at copy rate.)
constexpr u32 RECOVER_BATCH = 4;

__global__ void __launch_bounds__(BLOCK) k_recover_by_volume(u32 nv, u32 const* __restrict__ offs,
    u32 const* __restrict__ uses, UseDiv div, double const* __restrict__ sizes, u32 nc,
    double const* __restrict__ f, double* __restrict__ out)
{
  pdl_wait();
  u64 const t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  u32 const i = (u32)(t / nc), c = (u32)(t - (u64)i * nc);
  if (i >= nv) return;
  double sum = 0, size_sum = 0;
  u32 const e1 = offs[i + 1];
  u32 j = offs[i];
  for (; j + RECOVER_BATCH <= e1; j += RECOVER_BATCH) {
    u32 e[RECOVER_BATCH];
    double es[RECOVER_BATCH], fe[RECOVER_BATCH];
#pragma unroll
    for (u32 k = 0; k < RECOVER_BATCH; ++k) e[k] = use_high(div, uses[j + k]);
#pragma unroll
    for (u32 k = 0; k < RECOVER_BATCH; ++k) {
      es[k] = sizes[e[k]];
      fe[k] = f[(size_t)e[k] * nc + c];
    }
#pragma unroll
    for (u32 k = 0; k < RECOVER_BATCH; ++k) {
      size_sum += es[k];
      sum += es[k] * fe[k];
    }
  }
  for (; j < e1; ++j) {
    u32 const e = use_high(div, uses[j]);
    double const es = sizes[e];
    size_sum += es;
    sum += es * f[(size_t)e * nc + c];
  }
  out[t] = sum / size_sum;
}

__global__ void k_size_from_hessian(u32 nv, u32 nhc, double const* __restrict__ hess,
    double const* __restrict__ w, u32 nsol, double min_h, double max_h,
    double* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  double const* hs = hess + (size_t)i * nhc;
  double total = 0;
  for (u32 j = 0; j < nsol; ++j) {
    double norm = sqrt(dot_ref(hs, hs, 9));
    double hw = w ? w[j] : 1.0;
    total += hw * norm;
    hs += 9;
  }
  // clamp (size_from_hessian.cpp:34-40)
  double o = max_h - total;
  if (o < min_h) o = min_h;
  out[i] = o;
}

__global__ void k_axpy(u32 n, double a, double const* __restrict__ x,
    double const* __restrict__ y, double* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = a * x[i] + y[i];
}

template <u32 DIM>
__global__ void k_min_quality(u32 ne, u32 const* __restrict__ voe,
    double const* __restrict__ x, unsigned long long* minkey)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long key = ~0ull;
  if (i < ne) {
    double ex[4][3];
    load_corners<DIM>(voe, x, i, ex);
    key = order_key(elem_quality(DIM, ex, 1));
  }
  block_min_key(key, minkey);
}

}  // namespace

void element_gradients(Mesh& m, char const* name)
{
  cudaStream_t s = m.s;
  Tag* t = m.find_tag(0, name);
  if (!t || t->type != T_F64) throw Failure(E_ARG, std::string("no vertex field ") + name);
  u32 dim = m.dim, ne = m.count(dim), nc = t->ncomps;
  double* out = dalloc<double>((size_t)ne * nc * 3, s);
  if (ne) {
    u32 const* voe = m.ask_down(dim, 0);
    double const* f = static_cast<double const*>(t->data);
    // the components of a scalar and of its gradient, in 2D and 3D (the
    // size-field chain's); any other count goes a thread per element
    auto k = dim == 3 ? (nc == 1 ? k_element_gradients<3, 1> : nc == 3 ? k_element_gradients<3, 3> : nullptr)
           : dim == 2 ? (nc == 1 ? k_element_gradients<2, 1> : nc == 3 ? k_element_gradients<2, 3> : nullptr)
                      : nullptr;
    if (k)
      CK(launch_kernel(k, dim3(grid_for(ne, GRAD_BLOCK)), dim3(GRAD_BLOCK), 0, s, ne, voe,
          m.coords(), f, out));
    else
      CK(launch_kernel(k_element_gradients_any, dim3(grid_for(ne)), dim3(BLOCK), 0, s, dim, ne,
          voe, m.coords(), nc, f, out));
    CK_LAUNCH();
  }
  m.add_tag(dim, T_F64, (std::string("grad_") + name).c_str(), nc * 3, X_NOT, out);
}

void recover_by_volume(Mesh& m, char const* name)
{
  cudaStream_t s = m.s;
  u32 dim = m.dim;
  Tag* t = m.find_tag(dim, name);
  if (!t || t->type != T_F64) throw Failure(E_ARG, std::string("no element field ") + name);
  u32 nv = m.count(0), nc = t->ncomps;
  UpAdj const& ve = m.ask_up(0, dim, true);
  double* sizes = m.element_sizes();
  double* out = dalloc<double>((size_t)nv * nc, s);
  if (nv && nc) {
    CK(launch_kernel(k_recover_by_volume, dim3(grid_for((u64)nv * nc)), dim3(BLOCK), 0, s, nv, ve.offs,
        ve.uses, use_div(deg(dim, 0)), sizes, nc, static_cast<double const*>(m.find_tag(dim, name)->data), out));
    CK_LAUNCH();
  }
  dev_free(sizes, s);
  m.add_tag(0, T_F64, name, nc, X_NOT, out);
}

void size_from_hessian(Mesh& m, char const* hess_name, double const* weights, double min_h,
    double max_h)
{
  cudaStream_t s = m.s;
  Tag* t = m.find_tag(0, hess_name);
  if (!t || t->type != T_F64) throw Failure(E_ARG, std::string("no vertex field ") + hess_name);
  if (t->ncomps % 9 || !(max_h > min_h) || !(min_h > 0))
    throw Failure(E_ARG, "size_from_hessian needs 9k components and 0 < min_h < max_h");
  u32 nv = m.count(0), nsol = t->ncomps / 9;
  double* w = nullptr;
  if (weights) {
    for (u32 j = 0; j < nsol; ++j)
      if (!(weights[j] >= 0)) throw Failure(E_ARG, "negative Hessian weight");
    w = dalloc<double>(nsol, s);
    CK(cudaMemcpyAsync(w, weights, sizeof(double) * nsol, cudaMemcpyHostToDevice, s));
  }
  double* out = dalloc<double>(nv, s);
  if (nv) {
    CK(launch_kernel(k_size_from_hessian, dim3(grid_for(nv)), dim3(BLOCK), 0, s, nv, t->ncomps,
        static_cast<double const*>(t->data), w, nsol, min_h, max_h, out));
    CK_LAUNCH();
  }
  stream_sync(s);
  dev_free(w, s);
  m.add_tag(0, T_F64, "adapt_size", 1, X_NOT, out);
}

static double min_quality_of(Mesh& m, double const* x)
{
  cudaStream_t s = m.s;
  u32 ne = m.count(m.dim);
  unsigned long long* mk = reinterpret_cast<unsigned long long*>(m.mb->dev + 30);
  CK(cudaMemsetAsync(mk, 0xff, sizeof(unsigned long long), s));
  if (ne) {
    auto k = m.dim == 3 ? k_min_quality<3> : m.dim == 2 ? k_min_quality<2> : k_min_quality<1>;
    CK(launch_kernel(k, dim3(grid_for(ne)), dim3(BLOCK), 0, s, ne, m.ask_down(m.dim, 0), x, mk));
    CK_LAUNCH();
  }
  m.mb->fetch(s, 32);
  unsigned long long k;
  std::memcpy(&k, m.mb->host + 30, sizeof(k));
  return k == ~0ull ? DBL_MAX : from_order_key(k);
}

u32 warp_to_limit(Mesh& m, double qual_floor)
{
  cudaStream_t s = m.s;
  Tag* xt = m.find_tag(0, "coordinates");
  Tag* wt = m.find_tag(0, "warp");
  if (!xt || !wt || wt->ncomps != 3) throw Failure(E_ARG, "warp_to_limit needs a 3-vector warp");
  u32 n = m.count(0) * 3;
  double const* x = static_cast<double const*>(xt->data);
  double const* w = static_cast<double const*>(wt->data);
  double* xo = dalloc<double>(n, s);
  double factor = 1;
  u32 hit = 0;
  auto apply = [&]() {
    if (n) {
      CK(launch_kernel(k_axpy, dim3(grid_for(n)), dim3(BLOCK), 0, s, n, factor, w, x, xo));
      CK_LAUNCH();
    }
  };
  apply();
  // exceeds_limit (warp_to_limit.cpp:14-29); halving ends after at most
  // 64 steps, when the warp no longer moves any coordinate
  for (u32 it = 0; min_quality_of(m, xo) < qual_floor; ++it) {
    if (it >= 1100) throw Failure(E_NOCONVERGE, "warp_to_limit: quality floor not reached");
    hit = 1;
    factor /= 2;
    apply();
  }
  double* wo = dalloc<double>(n, s);
  if (n) {
    CK(launch_kernel(k_axpy, dim3(grid_for(n)), dim3(BLOCK), 0, s, n, -factor, w, w, wo));
    CK_LAUNCH();
  }
  m.remove_tag(0, "coordinates");
  m.remove_tag(0, "warp");
  m.add_tag(0, T_F64, "coordinates", 3, X_NOT, xo);
  m.add_tag(0, T_F64, "warp", 3, X_NOT, wo);
  dev_free(m.qual_cache, s);
  m.qual_cache = nullptr;
  return hit ? 0u : 1u;
}

}  // namespace osh
