// Ion density grids on the device (the reference's analysis/Mg_distribution_3D/
// calc_Mg_density.py, which histograms Mg positions read back from DCD frames
// fitted by bestfit_motifs.py): per frame, an optional least-squares superposition
// of selected beads onto reference coordinates, then every ion of one kind binned
// into a 3-D grid, all on the handle's stream with no host synchronisation.
#include "tis_kernels.cuh"

namespace tis {
namespace {

constexpr int kFitThreads = 256;

// Largest-eigenvalue eigenvector of the symmetric 4x4 matrix a (cyclic Jacobi
// rotations, at most 50 sweeps).
__device__ void eig4_max(double a[4][4], double q[4])
{
    double v[4][4] = {{1, 0, 0, 0}, {0, 1, 0, 0}, {0, 0, 1, 0}, {0, 0, 0, 1}};
    for (int sweep = 0; sweep < 50; ++sweep) {
        double off = 0.0;
        for (int i = 0; i < 4; ++i)
            for (int j = i + 1; j < 4; ++j) off += a[i][j] * a[i][j];
        if (off < 1e-300) break;
        for (int p = 0; p < 4; ++p)
            for (int r = p + 1; r < 4; ++r) {
                if (a[p][r] == 0.0) continue;
                const double th = 0.5 * (a[r][r] - a[p][p]) / a[p][r];
                const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
                for (int k = 0; k < 4; ++k) {  // a <- J^T a J
                    const double akp = a[k][p], akr = a[k][r];
                    a[k][p] = c * akp - s * akr;
                    a[k][r] = s * akp + c * akr;
                }
                for (int k = 0; k < 4; ++k) {
                    const double apk = a[p][k], ark = a[r][k];
                    a[p][k] = c * apk - s * ark;
                    a[r][k] = s * apk + c * ark;
                }
                for (int k = 0; k < 4; ++k) {
                    const double vkp = v[k][p], vkr = v[k][r];
                    v[k][p] = c * vkp - s * vkr;
                    v[k][r] = s * vkp + c * vkr;
                }
            }
    }
    int best = 0;
    for (int i = 1; i < 4; ++i)
        if (a[i][i] > a[best][best]) best = i;
    for (int k = 0; k < 4; ++k) q[k] = v[k][best];
}

// The same by Newton's method on det(a - l I) from an upper bound of its roots (the start
// Theobald takes, Acta Cryst. A 61, 478 (2005)), which descends to the largest one; d det/dl
// is minus the trace of the adjugate, whose columns at the root are the eigenvector.  Two
// iterations mostly, each one division deep, where the rotations chain four divisions and
// roots thirty times (with the rmsd summed by the block: a frame of 345 beads 490 -> 41 us with
// its launches).  False when the result is not an
// eigenvector to rounding (a near-double largest root, no correlation at all): the
// rotations decide then.
__device__ bool eig4_newton(const double (&a)[4][4], double bound, double q[4])
{
    double l = bound, c[4];
    double s0, s1, s2, s3, s4, s5, t0, t1, t2, t3, t4, t5, b00, b11, b22, b33;
    auto minors = [&]() {  // of rows 0, 1 and of rows 2, 3 of a - l I, over columns 01 02 03 12 13 23
        b00 = a[0][0] - l; b11 = a[1][1] - l; b22 = a[2][2] - l; b33 = a[3][3] - l;
        s0 = b00 * b11 - a[0][1] * a[1][0];
        s1 = b00 * a[1][2] - a[0][2] * a[1][0];
        s2 = b00 * a[1][3] - a[0][3] * a[1][0];
        s3 = a[0][1] * a[1][2] - a[0][2] * b11;
        s4 = a[0][1] * a[1][3] - a[0][3] * b11;
        s5 = a[0][2] * a[1][3] - a[0][3] * a[1][2];
        t0 = a[2][0] * a[3][1] - a[2][1] * a[3][0];
        t1 = a[2][0] * a[3][2] - b22 * a[3][0];
        t2 = a[2][0] * b33 - a[2][3] * a[3][0];
        t3 = a[2][1] * a[3][2] - b22 * a[3][1];
        t4 = a[2][1] * b33 - a[2][3] * a[3][1];
        t5 = b22 * b33 - a[2][3] * a[3][2];
        c[0] = b11 * t5 - a[1][2] * t4 + a[1][3] * t3;  // the adjugate's diagonal
        c[1] = b00 * t5 - a[0][2] * t2 + a[0][3] * t1;
        c[2] = a[3][0] * s4 - a[3][1] * s2 + b33 * s0;
        c[3] = a[2][0] * s3 - a[2][1] * s1 + b22 * s0;
    };
    for (int it = 0; it < 40; ++it) {
        minors();
        const double det = s0 * t5 - s1 * t4 + s2 * t3 + s3 * t2 - s4 * t1 + s5 * t0;
        const double step = det / (c[0] + c[1] + c[2] + c[3]);
        if (!(fabs(step) < 1e300)) return false;
        l += step;
        if (fabs(step) <= 1e-15 * fabs(l)) break;
    }
    minors();
    int j = 0;
    for (int k = 1; k < 4; ++k)
        if (fabs(c[k]) > fabs(c[j])) j = k;
    double v[4];  // column j of the adjugate
    if (j == 0) {
        v[0] = c[0];
        v[1] = -a[1][0] * t5 + a[1][2] * t2 - a[1][3] * t1;
        v[2] = a[1][0] * t4 - b11 * t2 + a[1][3] * t0;
        v[3] = -a[1][0] * t3 + b11 * t1 - a[1][2] * t0;
    } else if (j == 1) {
        v[0] = -a[0][1] * t5 + a[0][2] * t4 - a[0][3] * t3;
        v[1] = c[1];
        v[2] = -b00 * t4 + a[0][1] * t2 - a[0][3] * t0;
        v[3] = b00 * t3 - a[0][1] * t1 + a[0][2] * t0;
    } else if (j == 2) {
        v[0] = a[3][1] * s5 - a[3][2] * s4 + b33 * s3;
        v[1] = -a[3][0] * s5 + a[3][2] * s2 - b33 * s1;
        v[2] = c[2];
        v[3] = -a[3][0] * s3 + a[3][1] * s1 - a[3][2] * s0;
    } else {
        v[0] = -a[2][1] * s5 + b22 * s4 - a[2][3] * s3;
        v[1] = a[2][0] * s5 - b22 * s2 + a[2][3] * s1;
        v[2] = -a[2][0] * s4 + a[2][1] * s2 - a[2][3] * s0;
        v[3] = c[3];
    }
    const double n2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
    if (!(n2 > 0.0)) return false;
    const double inv = 1.0 / sqrt(n2);
    double r2 = 0.0, m2 = 0.0;
    for (int k = 0; k < 4; ++k) q[k] = v[k] * inv;
    for (int i = 0; i < 4; ++i) {
        double r = -l * q[i];
        for (int k = 0; k < 4; ++k) {
            r += a[i][k] * q[k];
            m2 += a[i][k] * a[i][k];
        }
        r2 += r * r;
    }
    return r2 <= 1e-29 * m2;  // residual within 3e-15 of the matrix
}

// One block: centroids and the correlation of the fit beads with their reference
// positions, then (one thread) the rotation of Horn's quaternion method (J. Opt.
// Soc. Am. A 4, 629 (1987)) taking the frame onto the reference:
// out = {R (9, row-major), frame centroid (3), reference centroid (3), rmsd}.
__global__ void __launch_bounds__(kFitThreads) k_fit(Dev d, int r, int n_fit, const int *idx, const double *ref,
                                                     double *out)
{
    __shared__ double s_red[17][kFitThreads / 32];
    const RepParams *R = d.rp + r;
    double acc[17] = {0};  // sums of x (3), of y (3), of x_a y_b (9), of |x|^2, of |y|^2
    for (int i = threadIdx.x; i < n_fit; i += blockDim.x) {
        const int p = R->p0 + idx[i];
        const double x[3] = {d.x[p], d.y[p], d.z[p]}, y[3] = {ref[3 * i], ref[3 * i + 1], ref[3 * i + 2]};
        for (int a = 0; a < 3; ++a) {
            acc[a] += x[a];
            acc[3 + a] += y[a];
            for (int b = 0; b < 3; ++b) acc[6 + 3 * a + b] += x[a] * y[b];
            acc[15] += x[a] * x[a];
            acc[16] += y[a] * y[a];
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 17; ++k) {
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], o);
        if (lane == 0) s_red[k][warp] = acc[k];
    }
    __shared__ double s_fit[15];  // rotation, frame centroid, reference centroid
    __syncthreads();
    const double inv = 1.0 / n_fit;
    __shared__ double s_sum[17];
    if (threadIdx.x < 17) {
        double v = 0.0;
        for (int w = 0; w < kFitThreads / 32; ++w) v += s_red[threadIdx.x][w];
        s_sum[threadIdx.x] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double *t = s_sum;
        const double xc[3] = {t[0] * inv, t[1] * inv, t[2] * inv}, yc[3] = {t[3] * inv, t[4] * inv, t[5] * inv};
        double S[3][3];  // sum (x - xc)_a (y - yc)_b
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) S[a][b] = t[6 + 3 * a + b] - n_fit * xc[a] * yc[b];
        double N[4][4] = {
            {S[0][0] + S[1][1] + S[2][2], S[1][2] - S[2][1], S[2][0] - S[0][2], S[0][1] - S[1][0]},
            {S[1][2] - S[2][1], S[0][0] - S[1][1] - S[2][2], S[0][1] + S[1][0], S[2][0] + S[0][2]},
            {S[2][0] - S[0][2], S[0][1] + S[1][0], -S[0][0] + S[1][1] - S[2][2], S[1][2] + S[2][1]},
            {S[0][1] - S[1][0], S[2][0] + S[0][2], S[1][2] + S[2][1], -S[0][0] - S[1][1] + S[2][2]}};
        // half the sum of both sets' squared radii bounds the largest eigenvalue
        double g = t[15] + t[16];
        for (int a = 0; a < 3; ++a) g -= n_fit * (xc[a] * xc[a] + yc[a] * yc[a]);
        double q[4];
        if (!eig4_newton(N, 0.5 * g * (1.0 + 1e-10), q)) eig4_max(N, q);
        const double q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
        const double Rm[9] = {q0 * q0 + q1 * q1 - q2 * q2 - q3 * q3, 2 * (q1 * q2 - q0 * q3), 2 * (q1 * q3 + q0 * q2),
                              2 * (q1 * q2 + q0 * q3), q0 * q0 - q1 * q1 + q2 * q2 - q3 * q3, 2 * (q2 * q3 - q0 * q1),
                              2 * (q1 * q3 - q0 * q2), 2 * (q2 * q3 + q0 * q1), q0 * q0 - q1 * q1 - q2 * q2 + q3 * q3};
        for (int k = 0; k < 9; ++k) s_fit[k] = Rm[k];
        for (int a = 0; a < 3; ++a) {
            s_fit[9 + a] = xc[a];
            s_fit[12 + a] = yc[a];
        }
    }
    __syncthreads();
    if (threadIdx.x < 15) out[threadIdx.x] = s_fit[threadIdx.x];
    double e2 = 0.0;  // rmsd after the fit, from the beads themselves
    for (int i = threadIdx.x; i < n_fit; i += blockDim.x) {
        const int p = R->p0 + idx[i];
        const double x[3] = {d.x[p] - s_fit[9], d.y[p] - s_fit[10], d.z[p] - s_fit[11]};
        for (int a = 0; a < 3; ++a) {
            const double v = s_fit[3 * a] * x[0] + s_fit[3 * a + 1] * x[1] + s_fit[3 * a + 2] * x[2] + s_fit[12 + a] - ref[3 * i + a];
            e2 += v * v;
        }
    }
    for (int o = 16; o > 0; o >>= 1) e2 += __shfl_down_sync(0xffffffffu, e2, o);
    if (lane == 0) s_red[0][warp] = e2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_red[0][w];
        out[15] = sqrt(t * inv);
    }
}

// every particle of replica r of `kind`: its (fitted) position binned into the grid
// lo + delta * [0, dims); the upper faces belong to the last bins (numpy.histogramdd)
__global__ void k_density(Dev d, int r, int kind, const double *fit, double lo0, double lo1, double lo2, double delta,
                          int nx, int ny, int nz, unsigned long long *grid)
{
    const RepParams *R = d.rp + r;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= R->n) return;
    const int p = R->p0 + i;
    if (((d.q[p].w >> 8) & 0xff) != kind) return;
    double x[3] = {d.x[p], d.y[p], d.z[p]};
    if (fit) {
        const double c[3] = {x[0] - fit[9], x[1] - fit[10], x[2] - fit[11]};
        for (int a = 0; a < 3; ++a) x[a] = fit[3 * a] * c[0] + fit[3 * a + 1] * c[1] + fit[3 * a + 2] * c[2] + fit[12 + a];
    }
    const double lo[3] = {lo0, lo1, lo2};
    const int dims[3] = {nx, ny, nz};
    int b[3];
    for (int a = 0; a < 3; ++a) {
        const double u = (x[a] - lo[a]) / delta;
        if (!(u >= 0.0) || u > (double)dims[a]) return;
        b[a] = min((int)floor(u), dims[a] - 1);
    }
    atomicAdd(grid + ((size_t)b[0] * ny + b[1]) * nz + b[2], 1ull);
}

}  // namespace

void launch_fit(const Dev &d, cudaStream_t s, int r, int n_fit, const int *idx, const double *ref, double *out)
{
    k_fit<<<1, kFitThreads, 0, s>>>(d, r, n_fit, idx, ref, out);
}

void launch_density(const Dev &d, cudaStream_t s, int r, int n, int kind, const double *fit, const double lo[3],
                    double delta, const int dims[3], unsigned long long *grid)
{
    k_density<<<(n + 255) / 256, 256, 0, s>>>(d, r, kind, fit, lo[0], lo[1], lo[2], delta, dims[0], dims[1], dims[2],
                                               grid);
}

}  // namespace tis
