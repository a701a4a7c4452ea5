// The division policies operand by operand, for test_gpu_division_operands.py: SharedDiv beside IeeeDiv on the
// same inputs.  `bad` is SharedDiv's flag: its results stand only where it is 0.
#include <cuda_runtime.h>

#include "awcm_numerics.cuh"

using namespace awcm;

__device__ long item() { return (long)blockIdx.x * blockDim.x + threadIdx.x; }

// out: quot, quot_pos, quotient by twice(b), recip, each by SharedDiv and by IeeeDiv
__global__ void k_quotients(const double* a, const double* b, long n, double* out)
{
    const long t = item();
    if (t >= n) return;
    SharedDiv s;
    IeeeDiv i;
    const auto d = s.by(b[t]);
    double* o = out + 8 * t;
    o[0] = s.quot(a[t], d), o[1] = i.quot(a[t], b[t]);
    o[2] = s.quot_pos(a[t], d), o[3] = i.quot_pos(a[t], b[t]);
    o[4] = s.quot(a[t], s.twice(d)), o[5] = i.quot(a[t], i.twice(b[t]));
    o[6] = s.recip(b[t]), o[7] = i.recip(b[t]);
}
// Bit 0: outside by range, bit 1: by range_or_0.
__global__ void k_ranges(const double* x, long n, int lo, int hi, int* out)
{
    const long t = item();
    if (t >= n) return;
    SharedDiv a, b;
    a.range(x[t], lo, hi);
    b.range_or_0(x[t], lo, hi);
    out[t] = (int)a.bad | (int)b.bad << 1;
}

template <class DV>
__device__ void all1(DV& face, DV& point, const double* q, double alpha, double g, int scheme, double* o)
{
    double s[6][3];
    for (int p = 0; p < 6; ++p)
        for (int k = 0; k < 3; ++k) s[p][k] = q[3 * p + k];
    if (scheme == kWeno5) face_flux_1d<kWeno5>(face, s, alpha, g, o);
    else face_flux_1d<kWenoZ>(face, s, alpha, g, o);
    o[3] = speed1(point, s[2][0], s[2][1], s[2][2], g);
    flux1(point, s[2], g, o + 4);
}
// out: flux[3], speed, physical flux[3], then the same by IeeeDiv; bad: of the face, of the point functions
__global__ void k_states1(const double* q, const double* alpha, const double* g, long n, int scheme, double* out, int* bad)
{
    const long t = item();
    if (t >= n) return;
    SharedDiv sf, sp;
    IeeeDiv i, j;
    all1(sf, sp, q + 18 * t, alpha[t], g[t], scheme, out + 14 * t);
    all1(i, j, q + 18 * t, alpha[t], g[t], scheme, out + 14 * t + 7);
    bad[2 * t] = sf.bad, bad[2 * t + 1] = sp.bad;
}

template <class DV>
__device__ void all2(DV& face, DV& point, const double* q, bool y, double alpha, double g, double eps, double delta, double* o)
{
    double s[6][4], prim[3];
    for (int p = 0; p < 6; ++p)
        for (int k = 0; k < 4; ++k) s[p][k] = q[4 * p + k];
    face_flux_2d(face, s, y, alpha, g, o, eps, delta);
    speeds2(point, s[2], g, o[4], o[5]);
    cell_flux2(point, s[2], g, o + 6, prim);
    for (int k = 0; k < 3; ++k) o[10 + k] = prim[k];
}
// out: flux[4], speeds[2], physical flux[4], primitives[3], then the same by IeeeDiv
__global__ void k_states2(const double* q, const double* alpha, const double* g, long n, int y, double eps, double delta,
                          double* out, int* bad)
{
    const long t = item();
    if (t >= n) return;
    SharedDiv sf, sp;
    IeeeDiv i, j;
    all2(sf, sp, q + 24 * t, y != 0, alpha[t], g[t], eps, delta, out + 26 * t);
    all2(i, j, q + 24 * t, y != 0, alpha[t], g[t], eps, delta, out + 26 * t + 13);
    bad[2 * t] = sf.bad, bad[2 * t + 1] = sp.bad;
}

static int done()
{
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
static unsigned blocks(long n) { return (unsigned)((n + 127) / 128); }

extern "C" {
int quotients(const double* a, const double* b, long n, double* out)
{
    k_quotients<<<blocks(n), 128>>>(a, b, n, out);
    return done();
}
int ranges(const double* x, long n, int lo, int hi, int* out)
{
    k_ranges<<<blocks(n), 128>>>(x, n, lo, hi, out);
    return done();
}
int states1(const double* q, const double* alpha, const double* g, long n, int scheme, double* out, int* bad)
{
    k_states1<<<blocks(n), 128>>>(q, alpha, g, n, scheme, out, bad);
    return done();
}
int states2(const double* q, const double* alpha, const double* g, long n, int y, double eps, double delta, double* out,
            int* bad)
{
    k_states2<<<blocks(n), 128>>>(q, alpha, g, n, y, eps, delta, out, bad);
    return done();
}
}
