// pose_chart.cu - VJP of the rigid chart pose = anchor exp(tangent^) with respect to the tangent.
//
// Replaces the reverse pass of the matrix exponential (python/dpt/torch/geometry.py:19-63
// differentiates torch.linalg.matrix_exp: an 8x8 exponential and some 90 launches, 1.2 ms of host
// time for two views) by the chart's own Jacobian in one launch.  With the body velocity (nu, phi)
// of exp(xi^) under a change of xi = (rho, omega), (nu, phi) = J(xi) (d rho, d omega) and
//   J = [[A, Q], [0, A]],  A = I - b1 W + a1 W^2,
//   Q = -P/2 + a1 (WP + PW - WPW) - a2 (WWP + PWW - 3 WPW) + a3 (WPWW + WWPW),
// W = omega^, P = rho^ (the right Jacobian of SE(3); Barfoot, State Estimation for Robotics,
// 7.1.5, with both arguments negated), a packed-pose cotangent G = (G_R, G_t) of the pose (R, t)
// gives f = R^T G_t, tau = axial part of R^T G_R and the tangent cotangent J^T (f, tau).
// One thread per view (nothing binds: a few hundred FP64 operations and one launch).
#include "launch.h"

namespace dpt {
namespace {

constexpr int kChartThreads = 128;

// Coefficients of the Jacobian at theta^2 = x.  Below theta = 2 their Taylor series in x (15
// terms: the last is below 1e-22 of the sum), above it the closed forms, whose cancellation is
// small there.
struct ChartCoefficients {
    double b1, a1, a2, a3;
    __device__ __forceinline__ explicit ChartCoefficients(double x)
    {
        if (x < 4.0) {
            // sum_k (-x)^k / (2k + 2)!, / (2k + 3)!, / (2k + 4)!, (k + 1) / (2k + 5)!, from the
            // last term: each factor is the ratio of two consecutive terms
            b1 = a1 = a2 = a3 = 1.0;
            for (int k = 14; k > 0; --k) {
                const double n = 2.0 * k;
                b1 = 1.0 - x / ((n + 1.0) * (n + 2.0)) * b1;
                a1 = 1.0 - x / ((n + 2.0) * (n + 3.0)) * a1;
                a2 = 1.0 - x / ((n + 3.0) * (n + 4.0)) * a2;
                a3 = 1.0 - x * ((k + 1.0) / k) / ((n + 4.0) * (n + 5.0)) * a3;
            }
            b1 /= 2.0;
            a1 /= 6.0;
            a2 /= 24.0;
            a3 /= 120.0;
        } else {
            const double t = sqrt(x);
            double s, c;
            sincos(t, &s, &c);
            b1 = (1.0 - c) / x;
            a1 = (t - s) / (x * t);
            a2 = (x + 2.0 * c - 2.0) / (2.0 * x * x);
            a3 = (2.0 * t - 3.0 * s + t * c) / (2.0 * x * x * t);
        }
    }
};

// r = a x b
__device__ __forceinline__ void cross3(const double* a, const double* b, double* r)
{
    r[0] = a[1] * b[2] - a[2] * b[1];
    r[1] = a[2] * b[0] - a[0] * b[2];
    r[2] = a[0] * b[1] - a[1] * b[0];
}

// J^T (f, tau) of one view.  The transposes apply W^T v = -omega x v, P^T v = -rho x v, so
//   A^T v = v + b1 (w x v) + a1 (w x (w x v)) and Q^T f likewise, right to left.
__device__ __forceinline__ void chart_vjp(const double* pose, const double* xi, const double* g, double* out)
{
    const double* rho = xi;
    const double* w = xi + 3;
    double m[9], f[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            m[3 * i + j] = pose[i] * g[j] + pose[3 + i] * g[3 + j] + pose[6 + i] * g[6 + j];
        f[i] = pose[i] * g[9] + pose[3 + i] * g[10] + pose[6 + i] * g[11];
    }
    const double tau[3] = {m[7] - m[5], m[2] - m[6], m[3] - m[1]};
    const ChartCoefficients k(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    double wf[3], wwf[3], pf[3], wt[3], wwt[3];
    cross3(w, f, wf);
    cross3(w, wf, wwf);
    cross3(rho, f, pf);
    cross3(w, tau, wt);
    cross3(w, wt, wwt);
    // words in X = w x, Y = rho x applied to f
    double xy[3], yx[3], xyx[3], xxy[3], yxx[3], xxyx[3], xyxx[3];
    cross3(w, pf, xy);
    cross3(rho, wf, yx);
    cross3(w, yx, xyx);
    cross3(w, xy, xxy);
    cross3(rho, wwf, yxx);
    cross3(w, xyx, xxyx);
    cross3(w, yxx, xyxx);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        out[i] = f[i] + k.b1 * wf[i] + k.a1 * wwf[i];
        const double q = 0.5 * pf[i] + k.a1 * (xy[i] + yx[i] + xyx[i]) + k.a2 * (xxy[i] + yxx[i] - 3.0 * xyx[i]) +
                         k.a3 * (xxyx[i] + xyxx[i]);
        out[3 + i] = q + tau[i] + k.b1 * wt[i] + k.a1 * wwt[i];
    }
}

// A tangent per view, one thread each.
__global__ void __launch_bounds__(kChartThreads) k_chart_vjp(int views, const double* __restrict__ poses,
                                                             const double* __restrict__ tangents,
                                                             const double* __restrict__ cotangents,
                                                             double* __restrict__ gradients)
{
    const int view = blockIdx.x * kChartThreads + threadIdx.x;
    if (view >= views) return;
    double out[6];
    chart_vjp(poses + 12 * (int64_t)view, tangents + 6 * (int64_t)view, cotangents + 12 * (int64_t)view, out);
#pragma unroll
    for (int i = 0; i < 6; ++i) gradients[6 * (int64_t)view + i] = out[i];
}

}  // namespace

cudaError_t launch_chart_vjp(int views, const double* poses, const double* tangents, const double* cotangents,
                             double* gradients, cudaStream_t stream)
{
    const unsigned blocks = (unsigned)(((int64_t)views + kChartThreads - 1) / kChartThreads);
    k_chart_vjp<<<blocks, kChartThreads, 0, stream>>>(views, poses, tangents, cotangents, gradients);
    return cudaGetLastError();
}

}  // namespace dpt

extern "C" int dpt_b200_pose_chart_vjp(int32_t views, const double* poses, const double* tangents,
                                       const double* cotangents, double* gradients, void* stream)
{
    if (!poses || !tangents || !cotangents || !gradients) return DPT_E_NULL;
    if (views < 1) return DPT_E_SHAPE;
    const cudaError_t error =
        dpt::launch_chart_vjp(views, poses, tangents, cotangents, gradients, static_cast<cudaStream_t>(stream));
    return error == cudaSuccess ? DPT_OK : (int)error;
}
