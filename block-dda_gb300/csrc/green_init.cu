// Green-tensor spectrum Ghat on the padded grid, built on the device in FP64.
//
// Replaces application_function + BT_fft + MBT_fft_init
// (mvp_fft/application_function.cpp:21-40, mvp_fft/BT_fft.cpp:8-53,
// mvp_fft/MBT_fft_init.cpp:22-35): instead of the length f^2 prod(2n_i-1) 1-D
// MBT projection, the 3x3 block A(d) = -G(d lf) is evaluated on the 2x-padded
// circulant grid (index j -> offset j for j < n, j - P for j > P - n, zero in
// the gap and at d = 0), its 6 distinct components (9 with the magnetic
// coupling of f = 6) are transformed once with the fixed-point core (mvp_fx.cu),
// divided by Px*Py*Pz and packed for each precision's z pass.
#include "mvp.hpp"

namespace bdda {

namespace {

__device__ __forceinline__ bool circ_offset(int j, int n, int P, int* d) {
  if (j < n) { *d = j; return true; }
  if (j > P - n) { *d = j - P; return true; }
  return false;
}

// g[comp][jx][jy][jz], comp = xx, xy, xz, yy, yz, zz of A = -G; with nc = 9
// (f = 6) also comp 6..8 = xy, xz, yz of B = -F, F = -k^2 e^{ikr}/r
// (1 - 1/(ikr)) [r^ x] (mvp_fft/application_function.cpp:52-64).
__global__ void k_green_eval(double2* __restrict__ g, int nc, int nx, int ny, int nz, int Px, int Py, int Pz,
                             double lf, double kr, double ki) {
  const size_t ng = (size_t)Px * Py * Pz;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < ng; idx += (size_t)gridDim.x * blockDim.x) {
    const int jz = (int)(idx % Pz);
    const int jy = (int)((idx / Pz) % Py);
    const int jx = (int)(idx / ((size_t)Pz * Py));
    int dx, dy, dz;
    double2 out[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) out[c] = make_double2(0.0, 0.0);
    if (circ_offset(jx, nx, Px, &dx) && circ_offset(jy, ny, Py, &dy) && circ_offset(jz, nz, Pz, &dz) &&
        (dx | dy | dz) != 0) {
      const double rx = dx * lf, ry = dy * lf, rz = dz * lf;
      const double r2 = rx * rx + ry * ry + rz * rz;
      const double r = sqrt(r2);
      // e = exp(i k r) / r with complex k = kr + i ki
      double sn, cs;
      sincos(kr * r, &sn, &cs);
      const double damp = exp(-ki * r) / r;
      const double2 e = make_double2(damp * cs, damp * sn);
      // c1 = k^2 ; c2 = (1 - i k r) / r^2
      const double2 c1 = make_double2(kr * kr - ki * ki, 2.0 * kr * ki);
      const double2 c2 = make_double2((1.0 + ki * r) / r2, (-kr * r) / r2);
      const double u[3] = {rx, ry, rz};
      int c = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = a; b < 3; ++b) {
          const double rr = u[a] * u[b] / r2;
          const double dl = (a == b) ? 1.0 : 0.0;
          // G_ab = (c1 (d - rr) - c2 (d - 3 rr)) e ; A = -G
          const double p = dl - rr, q = dl - 3.0 * rr;
          const double2 t = make_double2(c1.x * p - c2.x * q, c1.y * p - c2.y * q);
          const double2 gab = cmul(t, e);
          out[c++] = make_double2(-gab.x, -gab.y);
        }
      }
      if (nc == 9) {
        // fac = -k^2 e (1 - 1/w), w = i k r; B = -F: B_xy = fac u_z, B_xz = -fac u_y, B_yz = fac u_x
        const double2 w = make_double2(-ki * r, kr * r);
        const double w2 = w.x * w.x + w.y * w.y;
        const double2 one_m = make_double2(1.0 - w.x / w2, w.y / w2);  // 1 - conj(w) / |w|^2
        const double2 ce = cmul(c1, e);
        const double2 fac = cmul(make_double2(-ce.x, -ce.y), one_m);
        const double ux = rx / r, uy = ry / r, uz = rz / r;
        out[6] = make_double2(fac.x * uz, fac.y * uz);
        out[7] = make_double2(-fac.x * uy, -fac.y * uy);
        out[8] = make_double2(fac.x * ux, fac.y * ux);
      }
    }
    for (int c = 0; c < nc; ++c) g[(size_t)c * ng + idx] = out[c];
  }
}

// g[comp][fixed-point order] * scale -> ghat[qx][qy][comp][green_pos(qz)] in
// complex FP32, qx / qy / qz in the complex FP32 plans' order (pos: its
// positions in the fixed-point order; rl = 0: natural order along z, else
// last-radix-major, see green_perm_radix)
__global__ void k_green_pack(const double2* __restrict__ g, float2* __restrict__ out, const int* __restrict__ pos, int nc,
                             int Px, int Py, int Pz, double scale, int rl) {
  const size_t ng = (size_t)Px * Py * Pz;
  const size_t total = (size_t)nc * ng;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int qz = (int)(idx % Pz);
    const size_t t = idx / Pz;
    const int comp = (int)(t % nc);
    const int line = (int)(t / nc);  // qx * Py + qy
    const int qx = line / Py, qy = line - qx * Py;
    const size_t src = ((size_t)pos[qx] * Py + pos[kMaxLine + qy]) * Pz + pos[2 * kMaxLine + qz];
    const double2 v = g[(size_t)comp * ng + src];
    out[idx - qz + green_pos(qz, Pz, rl)] = make_float2((float)(v.x * scale), (float)(v.y * scale));
  }
}

}  // namespace

cudaError_t build_green_hat(const MvpGeom& g, double lf, double k_re, double k_im, const FxTables& t, double2* work,
                            float2* ghat_f, const int* pos, fx::Fac* ghat_x, int* gexp, cudaStream_t st) {
  const int Px = g.Px, Py = g.Py, Pz = g.Pz;
  const size_t ng = (size_t)Px * Py * Pz;
  const int nc = g.f == 6 ? 9 : 6;
  k_green_eval<<<1216, 256, 0, st>>>(work, nc, g.nx, g.ny, g.nz, Px, Py, Pz, lf, k_re, k_im);
  cudaError_t e = fx_green_transform(work, nc, t, st);
  if (e != cudaSuccess) return e;
  const double scale = 1.0 / (double)ng;
  if (ghat_x) {
    e = fx_green_pack(work, nc, t, ghat_x, gexp, scale, st);
    if (e != cudaSuccess) return e;
  }
  if (ghat_f) k_green_pack<<<2432, 256, 0, st>>>(work, ghat_f, pos, nc, Px, Py, Pz, scale, g.gperm);
  return cudaGetLastError();
}

}  // namespace bdda
