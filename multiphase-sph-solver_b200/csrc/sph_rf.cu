// sph_rf.cu -- the correlation-matrix random fields on the device
// (clFSpatialVariability_Fun::nonstationary_random_2D / _3D,
// CPP_17-3-Nonstationary-RF.cpp:76-849, flspv 3; and
// nonstationary_correlated_random_2D / _3D,
// CPP_17-5-Nonstationary-Correlated-RF.cpp:87-735, flspv 4).
//
// The reference divides the widened non-boundary box into cells of cell_ndx
// spacings, forms the correlation matrix of the cell centres, factors it by a
// row-oriented Cholesky with the diagonal's radicand floored at 1e-6,
// multiplies the factor by standard normals and gives every particle of a
// cell the cell's value.  Here every stage runs on the GPU:
//   k_rf_cells   the cell of each particle and the per-cell counts (a cell of
//                more than 39 particles is the reference's error 42)
//   k_rf_corr    the correlation matrix's lower triangle, one thread per entry
//   k_rf_panel   a 64-column panel: its diagonal block factored, the rows below
//                solved against it
//   k_rf_update  the trailing lower triangle less the panel's outer product
//                (64 x 64 output tiles)
//   k_rf_gemv    E = L zeta, one warp per row
//   k_rf_assign  each particle's value from its cell (normal or lognormal map
//                with the depth trend, as the reference writes it)
// The blocked factorisation adds its products in another order than the
// reference's row sums, so values agree to rounding, not bit for bit.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#define RF_B 64
#define RF_MAXP 39

namespace {

struct RFArgs {
    int ndim, n, no, type, flag_auto;
    int depth_axis;          // the centre coordinate the depth trend reads
    int log_exp;             // lognormal map as exp(.) (1) or pow(e, .) (0)
    int nc[3], total;
    double base[3], cdx, dr;
    double mean_value, sd_value, coe_depth, rl[3], beta, beta1, soil_max, water_max;
};

__device__ __forceinline__ void centre(const RFArgs& a, int c, double x[3])
{
    const int i = c % a.nc[0], j = (c / a.nc[0]) % a.nc[1], k = c / (a.nc[0] * a.nc[1]);
    x[0] = a.base[0] + ((double)i + 0.5) * a.cdx;
    x[1] = a.base[1] + ((double)j + 0.5) * a.cdx;
    x[2] = (a.ndim == 3) ? a.base[2] + ((double)k + 0.5) * a.cdx : 0.0;
}

__global__ void k_rf_cells(RFArgs a, const double* xh, const int* type, int* cell, int* count, int* err)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    cell[i] = -1;
    if (a.ndim == 2 && !(type[i] == 1 || type[i] == 2)) return;
    const double* p = xh + 4 * (size_t)i;
    int np[3] = {0, 0, 0};
    for (int d = 0; d < a.ndim; d++) np[d] = (int)(fabs(p[d] - a.base[d]) / a.cdx);
    for (int d = 0; d < a.ndim; d++)
        if (np[d] < 0 || np[d] >= a.nc[d]) { err[0] = 1; return; }
    const int c = (a.ndim == 2) ? np[1] * a.nc[0] + np[0] : np[2] * a.nc[0] * a.nc[1] + np[1] * a.nc[0] + np[0];
    if (atomicAdd(&count[c], 1) >= RF_MAXP) err[1] = 1;
    cell[i] = c;
}

// the autocorrelation of two cell centres (CPP_17-3:210-224, 600-616)
__global__ void k_rf_corr(RFArgs a, double* C)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (j > k) return;                       // the factorisation reads the lower triangle
    double xk[3], xj[3];
    centre(a, k, xk);
    centre(a, j, xj);
    const double dx = fabs(xk[0] - xj[0]), dy = fabs(xk[1] - xj[1]);
    const double pi = 3.141592653;
    double acf;
    if (a.ndim == 2) {
        if (a.flag_auto == 1) acf = exp(-2.0 * (dx / a.rl[0] + dy / a.rl[1]));
        else if (a.flag_auto == 2) acf = exp(-pi * (pow(dx / a.rl[0], 2.0) + pow(dy / a.rl[1], 2.0)));
        else acf = exp(-2.0 * ((dx * cos(a.beta) + dy * sin(a.beta)) / a.rl[0] +
                               (-dx * sin(a.beta) + dy * cos(a.beta)) / a.rl[1]));
    } else {
        const double dz = fabs(xk[2] - xj[2]);
        const double t0 = dx * cos(a.beta1) + dy * sin(a.beta1);
        const double t1 = (-dx * sin(a.beta1) + dy * cos(a.beta1)) * cos(a.beta) + dz * sin(a.beta);
        const double t2 = -(-dx * sin(a.beta1) + dy * cos(a.beta1)) * sin(a.beta) + dz * cos(a.beta);
        if (a.flag_auto == 1) acf = exp(-2.0 * (dx / a.rl[0] + dy / a.rl[1] + dz / a.rl[2]));
        else if (a.flag_auto == 2)
            acf = exp(-pi * (pow(dx / a.rl[0], 2.0) + pow(dy / a.rl[1], 2.0) + pow(dz / a.rl[2], 2.0)));
        else acf = exp(-2.0 * (t0 / a.rl[0] + t1 / a.rl[1] + t2 / a.rl[2]));
    }
    C[(size_t)k * a.total + j] = acf;
}

// A panel: the diagonal block [k0, k0 + 64) factored (right-looking, the
// radicand floored at 1e-6), and L[i][k0 .. k0 + 64) for the 64 rows below that
// the block takes, by forward substitution.  Every block factors the diagonal
// block for itself, in place of a launch of one block that the others wait
// for.  Four threads hold a row, every fourth column each, in registers: a
// step of either part is one column's quotients, then the multiply-adds of all
// later columns, which are independent (a running sum per column is a chain of
// 2,016).  Quotients by the pivot are taken from its reciprocal with one
// correction step.  The factored block goes to `diag`, from where k_rf_update
// puts it into the matrix (other blocks may still be reading the unfactored
// one here).  Rows and columns past n read as the identity's.  Bound by
// latency: 64 steps of a reciprocal root and two barriers, then 64 of a
// broadcast and a quotient: 36 us a panel (45 with a square root and a
// reciprocal each; 130 with one thread per row).
// (An infinite x, as rotated kernels of short correlation lengths give, leaves
// no finite residual: its quotient is the product.)
__device__ __forceinline__ double rf_quotient(double x, double y, double ry)
{
    const double q = x * ry, r = fma(-q, y, x);
    return isfinite(r) ? fma(r, ry, q) : q;
}

__global__ void __launch_bounds__(4 * RF_B) k_rf_panel(double* A, double* diag, int n, int k0)
{
    __shared__ double lt[RF_B][RF_B + 2];            // the factor, column by column
    __shared__ double raw[2][RF_B];                  // the next column before its division, by turns
    __shared__ double rec[RF_B];                     // the pivots' reciprocals
    const int t = threadIdx.x, row = t >> 2, q = t & 3, lane = t & 31;
    constexpr int U = RF_B / 4;
    double x[U];                                     // columns 4 u + q
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int j = 4 * u + q;
        const bool in = k0 + row < n && k0 + j < n;
        x[u] = (in && j <= row) ? A[(size_t)(k0 + row) * n + k0 + j] : (j == row) ? 1.0 : 0.0;
    }
    if (q == 0) raw[0][row] = x[0];
#pragma unroll
    for (int k = 0; k < RF_B; k++) {
        __syncthreads();
        // the pivot's root and its reciprocal from one reciprocal root
        const double v = raw[k & 1][k], f = v > 1.0e-6 ? v : 1.0e-6, r = rsqrt(f), p0 = f * r;
        const double p = fma(fma(-p0, p0, f), 0.5 * r, p0);
        const double l = (row == k) ? p : (row > k) ? rf_quotient(raw[k & 1][row], p, r) : 0.0;
        if (q == 0) {
            lt[k][row] = l;
            if (row == k) rec[k] = r;
        }
        __syncthreads();
#pragma unroll
        for (int u = (k + 1) / 4; u < U; u++) x[u] = fma(-l, lt[k][4 * u + q], x[u]);   // (columns up to k: unused)
        if (k + 1 < RF_B && q == ((k + 1) & 3)) raw[(k + 1) & 1][row] = x[(k + 1) / 4];
    }
    __syncthreads();
    if (blockIdx.x == 0)
        for (int e = t; e < RF_B * RF_B; e += 4 * RF_B) diag[e] = lt[e % RF_B][e / RF_B];
    const int i = k0 + RF_B + blockIdx.x * RF_B + row;
    if (k0 + RF_B >= n) {
        // the last panel: one block, nobody else reads the matrix
        for (int e = t; e < RF_B * RF_B; e += 4 * RF_B) {
            const int a = e / RF_B, b = e % RF_B;
            if (b <= a && k0 + a < n) A[(size_t)(k0 + a) * n + k0 + b] = lt[b][a];
        }
        return;
    }
    const double* src = A + (size_t)min(i, n - 1) * n + k0 + q;
#pragma unroll
    for (int u = 0; u < U; u++) x[u] = src[4 * u];
#pragma unroll
    for (int k = 0; k < RF_B; k++) {
        const double mine = __shfl_sync(0xffffffffu, x[k / 4], (lane & ~3) | (k & 3));
        const double xk = rf_quotient(mine, lt[k][k], rec[k]);
        if (q == (k & 3)) x[k / 4] = xk;
#pragma unroll
        for (int u = k / 4; u < U; u++)
            if (4 * u + q > k) x[u] = fma(-xk, lt[k][4 * u + q], x[u]);
    }
    if (i < n)
#pragma unroll
        for (int u = 0; u < U; u++) A[(size_t)i * n + k0 + q + 4 * u] = x[u];
}

// the trailing lower triangle, A[i][j] -= sum_k L[i][k] L[j][k] over the
// panel's 64 columns, for k0 + 64 <= j <= i < n: 64 x 64 output tiles, the
// panel's columns staged 16 at a time (k-major, one column of padding so the
// transposing stores fall in distinct banks); each thread owns rows
// tr + 16 p and columns tc + 16 q, so the tile reads and writes are 128-byte
// runs, and sums its products from zero: the small products' sum, subtracted
// once, loses less.  Multiply-adds on registers: on the FP64 tensor cores
// (mma.sync m8n8k4, whole panels staged) one update of 2,366, 4,766 and 13,184
// rows takes 40, 137 and 849 us, here 33, 104 and 707 (15.8 TFLOP/s; a factor of
// 13,248 cells 68.5 -> 58.4 ms).  The width bs (64) stays an argument: with the
// loop's count known, ptxas schedules it into 41, 112 and 850.
__global__ void __launch_bounds__(256) k_rf_update(double* A, const double* diag, int n, int k0, int bs)
{
    if (blockIdx.x == 0)
        for (int e = threadIdx.x; e < RF_B * RF_B; e += 256)
            if (e % RF_B <= e / RF_B) A[(size_t)(k0 + e / RF_B) * n + k0 + e % RF_B] = diag[e];

    // tile (r, c), c <= r, of the trailing triangle, numbered row by row
    int r = (int)((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= (int)blockIdx.x) r++;
    while (r * (r + 1) / 2 > (int)blockIdx.x) r--;
    const int c = blockIdx.x - r * (r + 1) / 2;
    const int r0 = k0 + RF_B + r * RF_B, c0 = k0 + RF_B + c * RF_B;
    __shared__ double As[16][RF_B + 1], Bs[16][RF_B + 1];
    const int tr = threadIdx.x / 16, tc = threadIdx.x % 16;
    double acc[4][4];
    for (int p = 0; p < 4; p++)
        for (int q = 0; q < 4; q++) acc[p][q] = 0.0;
    for (int kc = 0; kc < bs; kc += 16) {
        __syncthreads();
        for (int e = threadIdx.x; e < 16 * RF_B; e += 256) {
            const int k = e % 16, x = e / 16;
            const bool in = kc + k < bs;
            As[k][x] = (in && r0 + x < n) ? A[(size_t)(r0 + x) * n + k0 + kc + k] : 0.0;
            Bs[k][x] = (in && c0 + x < n) ? A[(size_t)(c0 + x) * n + k0 + kc + k] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) {
            double a[4], b[4];
#pragma unroll
            for (int p = 0; p < 4; p++) { a[p] = As[k][tr + 16 * p]; b[p] = Bs[k][tc + 16 * p]; }
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[p][q] = fma(a[p], b[q], acc[p][q]);
        }
    }
    for (int p = 0; p < 4; p++)
        for (int q = 0; q < 4; q++) {
            const int i = r0 + tr + 16 * p, j = c0 + tc + 16 * q;
            if (i < n && j <= i) A[(size_t)i * n + j] = A[(size_t)i * n + j] - acc[p][q];
        }
}

// E = L zeta over the lower triangle, one warp per row
__global__ void k_rf_gemv(const double* L, int n, const double* zeta, double* E)
{
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= n) return;
    double t = 0.0;
    for (int j = lane; j <= row; j += 32) t = t + L[(size_t)row * n + j] * zeta[j];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) E[row] = t;
}

// each particle's value (CPP_17-3:235-450, 17-5:222-402): its cell's normal
// value with the depth trend from soil_max (soil members) or water_max (fluid
// members), or the lognormal map with the trend from soil_max for every
// member, as the reference writes them.  The depth is the centre's last
// coordinate, except for the fluid members of the correlated 3-D field, which
// read y (17-5:655-735); the correlated field maps lognormals through exp,
// the single field through pow(e, .).
__global__ void k_rf_assign(RFArgs a, const int* cell, const int* type, const double* E, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int c = cell[i];
    const bool soil = a.no <= 3;
    double v = __longlong_as_double(0x7ff8000000000000LL);
    if (c >= 0 && type[i] == (soil ? 2 : 1)) {
        double x[3];
        centre(a, c, x);
        const double depth = x[a.depth_axis];
        if (a.type == 1) {
            const double top = soil ? a.soil_max : a.water_max;
            if (top > depth) v = a.mean_value + a.coe_depth * (top - depth) + a.sd_value * E[c];
            else v = a.mean_value + a.sd_value * E[c];
        } else {
            double m = (a.soil_max > depth) ? a.mean_value + a.coe_depth * (a.soil_max - depth) : a.mean_value;
            const double sd = sqrt(log(1.0 + (a.sd_value / m) * (a.sd_value / m)));
            m = log(m) - 0.5 * sd * sd;
            v = a.log_exp ? exp(m + sd * E[c]) : pow(exp(1.0), m + sd * E[c]);
        }
    }
    out[i] = v;
}

RFArgs rf_args(const int* ip, const double* dp)
{
    RFArgs a;
    a.ndim = ip[0]; a.n = ip[1]; a.no = ip[2]; a.type = ip[3]; a.flag_auto = ip[4];
    for (int d = 0; d < 3; d++) { a.nc[d] = ip[5 + d]; a.base[d] = dp[d]; a.rl[d] = dp[3 + d]; }
    a.depth_axis = ip[8]; a.log_exp = ip[9];
    a.total = a.nc[0] * a.nc[1] * a.nc[2];
    a.cdx = dp[6]; a.dr = dp[7];
    a.mean_value = dp[8]; a.sd_value = dp[9]; a.coe_depth = dp[10];
    a.beta = dp[11]; a.beta1 = dp[12]; a.soil_max = dp[13]; a.water_max = dp[14];
    return a;
}

}  // namespace

// The host passes the field's description as two arrays:
//   ip: ndim, n, no, type, flag_auto, nc[3], depth axis, lognormal form
//   dp: base[3], rl[3], cell edge, dr, mean, sd, coe_depth, beta, beta_1
//       (radians), soil_max, water_max
// Positions are (x, y, z, h) records, 4 doubles per particle.

// Stage 1: the cell of each particle (-1 for none) and the per-cell counts
// (d_count zeroed by the caller); d_err[0] is set for a particle outside the
// cells, d_err[1] for a cell of more than 39 particles (d_err zeroed).
extern "C" int sphk_rf_cells(const int* ip, const double* dp, const double* d_xh, const int* d_type, int* d_cell,
                             int* d_count, int* d_err, cudaStream_t st)
{
    const RFArgs a = rf_args(ip, dp);
    if (a.n > 0) k_rf_cells<<<(a.n + 255) / 256, 256, 0, st>>>(a, d_xh, d_type, d_cell, d_count, d_err);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// Stage 2: the correlation matrix of the cell centres into d_C (total x
// total, row-major) and its lower Cholesky factor in place (the entries above
// the diagonal are left undefined).  d_C has room for sphk_rf_matrix_doubles.
extern "C" size_t sphk_rf_matrix_doubles(size_t total) { return total * total + RF_B * RF_B; }

extern "C" int sphk_rf_factor(const int* ip, const double* dp, double* d_C, cudaStream_t st)
{
    const RFArgs a = rf_args(ip, dp);
    const int T = a.total;
    k_rf_corr<<<dim3((T + 255) / 256, T), 256, 0, st>>>(a, d_C);
    double* d_diag = d_C + (size_t)T * T;
    for (int k0 = 0; k0 < T; k0 += RF_B) {
        const int rest = T - k0 - RF_B;
        const int tiles = (rest > 0) ? (rest + RF_B - 1) / RF_B : 0;
        k_rf_panel<<<tiles > 0 ? tiles : 1, 4 * RF_B, 0, st>>>(d_C, d_diag, T, k0);
        if (tiles > 0) k_rf_update<<<tiles * (tiles + 1) / 2, 256, 0, st>>>(d_C, d_diag, T, k0, RF_B);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// Stage 3: E = L zeta and each particle's value into d_out (NaN where the
// field writes none).
extern "C" int sphk_rf_assign(const int* ip, const double* dp, const double* d_L, const double* d_zeta, double* d_E,
                              const int* d_cell, const int* d_type, double* d_out, cudaStream_t st)
{
    const RFArgs a = rf_args(ip, dp);
    const int T = a.total;
    k_rf_gemv<<<(T * 32 + 255) / 256, 256, 0, st>>>(d_L, T, d_zeta, d_E);
    if (a.n > 0) k_rf_assign<<<(a.n + 255) / 256, 256, 0, st>>>(a, d_cell, d_type, d_E, d_out);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
