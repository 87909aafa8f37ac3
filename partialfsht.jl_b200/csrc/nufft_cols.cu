// The NUFFT's column stages in one kernel each way, FP64: the FFT along Theta of a mode column, the
// per-mode factors and zero padding, the fine FFT along dim 1 and the transpose of the kept rows
// into U (type 2), and their transpose (type 1). The library chain is four kernels (Theta FFT, pad,
// FFT, rows) that pass the padded columns through memory three times; below a few million fine
// cells each of them is mostly its launch (6-8 us each of 109 us a pass at lmax 256).
//
// A block takes C neighbouring columns through shared memory: Stockham passes of radix 2 to 9
// between two buffers of C columns (a thread per butterfly, the twiddles from a table of the
// length's roots of unity), so a block has about seven barriers for the two transforms, and
// writes the kept rows with C neighbouring fine columns together. Lengths whose columns do not fit
// twice into shared memory, or with a prime factor over 7, keep the library chain.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"

namespace pf {

namespace {

constexpr int kMaxThreads = 256;
constexpr size_t kMaxSmem = 100 * 1024;

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a times s i (s = +-1)
__device__ __forceinline__ double2 cimul(double2 a, double s) { return make_double2(-s * a.y, s * a.x); }

// in-place DFTs of R values with exponent sign s
template <int R> struct Dft;
template <> struct Dft<2> {
    __device__ static void run(double2 (&v)[2], double) {
        const double2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    }
};
template <> struct Dft<3> {
    __device__ static void run(double2 (&v)[3], double s) {
        const double h = 0.86602540378443864676;
        const double2 t = cadd(v[1], v[2]), d = cimul(csub(v[1], v[2]), s * h);
        const double2 m = make_double2(fma(-0.5, t.x, v[0].x), fma(-0.5, t.y, v[0].y));
        v[0] = cadd(v[0], t);
        v[1] = cadd(m, d);
        v[2] = csub(m, d);
    }
};
template <> struct Dft<4> {
    __device__ static void run(double2 (&v)[4], double s) {
        const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = cimul(csub(v[1], v[3]), s);
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    }
};
template <> struct Dft<5> {
    __device__ static void run(double2 (&v)[5], double s) {
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
        const double2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
        const double2 a = make_double2(v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y);
        const double2 b = make_double2(v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y);
        const double2 e = cimul(make_double2(s1 * d1.x + s2 * d2.x, s1 * d1.y + s2 * d2.y), s);
        const double2 f = cimul(make_double2(s2 * d1.x - s1 * d2.x, s2 * d1.y - s1 * d2.y), s);
        v[0] = cadd(v[0], cadd(t1, t2));
        v[1] = cadd(a, e);
        v[2] = cadd(b, f);
        v[3] = csub(b, f);
        v[4] = csub(a, e);
    }
};
template <> struct Dft<7> {
    __device__ static void run(double2 (&v)[7], double s) {
        const double c[3] = {0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
        const double sn[3] = {0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
        double2 t[3], d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            t[k] = cadd(v[1 + k], v[6 - k]);
            d[k] = csub(v[1 + k], v[6 - k]);
        }
        double2 out[7];
        out[0] = cadd(v[0], cadd(t[0], cadd(t[1], t[2])));
#pragma unroll
        for (int j = 1; j <= 3; ++j) {
            double2 a = v[0], e = make_double2(0.0, 0.0);
#pragma unroll
            for (int k = 1; k <= 3; ++k) {
                const int p = (j * k) % 7;  // cos and sin of 2 pi p / 7 from the first three
                const double cc = c[(p <= 3 ? p : 7 - p) - 1], ss = p <= 3 ? sn[p - 1] : -sn[6 - p];
                a.x = fma(cc, t[k - 1].x, a.x);
                a.y = fma(cc, t[k - 1].y, a.y);
                e.x = fma(ss, d[k - 1].x, e.x);
                e.y = fma(ss, d[k - 1].y, e.y);
            }
            const double2 f = cimul(e, s);
            out[j] = cadd(a, f);
            out[7 - j] = csub(a, f);
        }
#pragma unroll
        for (int j = 0; j < 7; ++j) v[j] = out[j];
    }
};
template <> struct Dft<8> {
    __device__ static void run(double2 (&v)[8], double s) {
        const double h = 0.70710678118654752440;
        double2 a[4] = {v[0], v[2], v[4], v[6]}, b[4] = {v[1], v[3], v[5], v[7]};
        Dft<4>::run(a, s);
        Dft<4>::run(b, s);
        // times e^{s i pi k / 4}
        b[1] = make_double2(h * (b[1].x - s * b[1].y), h * (b[1].y + s * b[1].x));
        b[2] = cimul(b[2], s);
        b[3] = make_double2(-h * (b[3].x + s * b[3].y), h * (s * b[3].x - b[3].y));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = cadd(a[k], b[k]);
            v[k + 4] = csub(a[k], b[k]);
        }
    }
};
template <> struct Dft<9> {
    __device__ static void run(double2 (&v)[9], double s) {
        // e^{s 2 pi i k / 9}, k = 1, 2, 4
        const double2 w1 = make_double2(0.76604444311897803520, s * 0.64278760968653932632);
        const double2 w2 = make_double2(0.17364817766693034885, s * 0.98480775301220805937);
        const double2 w4 = make_double2(-0.93969262078590838405, s * 0.34202014332566873304);
        double2 u[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            u[j][0] = v[j];
            u[j][1] = v[j + 3];
            u[j][2] = v[j + 6];
            Dft<3>::run(u[j], s);
        }
        u[1][1] = cmul(u[1][1], w1);
        u[1][2] = cmul(u[1][2], w2);
        u[2][1] = cmul(u[2][1], w2);
        u[2][2] = cmul(u[2][2], w4);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double2 x[3] = {u[0][k], u[1][k], u[2][k]};
            Dft<3>::run(x, s);
            v[k] = x[0];
            v[k + 3] = x[1];
            v[k + 6] = x[2];
        }
    }
};

// i / d for i, d < 2^16 by multiplication
struct Div {
    unsigned d, mul;
};
__device__ __forceinline__ unsigned quot(unsigned i, Div d) { return d.d == 1 ? i : __umulhi(i, d.mul); }

// one pass of C transforms of length n between two buffers (columns n apart): radix R, ns the product
// of the radices before it
template <int R>
__device__ __forceinline__ void pass(const double2* in, double2* out, int n, int C, Div per, Div ns, double s,
                                     const double2* __restrict__ roots) {
    const int m = (int)per.d;  // butterflies of one transform, n / R
    const int step = m / (int)ns.d;
    for (int i = threadIdx.x; i < C * m; i += blockDim.x) {
        const int c = (int)quot(i, per), j = i - c * m;
        const int h = (int)quot(j, ns), k = j - h * (int)ns.d;
        const double2* p = in + c * n + j;
        double2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = p[q * m];
        if (k > 0) {
#pragma unroll
            for (int q = 1; q < R; ++q) {
                double2 w = roots[q * k * step];
                w.y *= s;
                v[q] = cmul(v[q], w);
            }
        }
        Dft<R>::run(v, s);
        double2* o = out + c * n + h * (int)ns.d * R + k;
#pragma unroll
        for (int q = 0; q < R; ++q) o[q * (int)ns.d] = v[q];
    }
}

struct Fft {
    int n = 0, npass = 0;
    int radix[12];
    Div per[12], ns[12];
};

// C transforms from buffer a to buffer a or b; returns where they end. Ends with a barrier.
__device__ __forceinline__ double2* fft(double2* a, double2* b, const Fft& f, int C, double s,
                                        const double2* __restrict__ roots) {
    for (int p = 0; p < f.npass; ++p) {
        switch (f.radix[p]) {
            case 2: pass<2>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
            case 3: pass<3>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
            case 4: pass<4>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
            case 5: pass<5>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
            case 7: pass<7>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
            case 8: pass<8>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
            default: pass<9>(a, b, f.n, C, f.per[p], f.ns[p], s, roots); break;
        }
        __syncthreads();
        double2* t = a;
        a = b;
        b = t;
    }
    return a;
}

struct Cols {
    Fft th, f1;            // along Theta (n1 modes) and along the fine columns (nf1)
    int ncols, row0, nrows, nf2, gap_lo, gap_hi;
    int C, nblocks;        // columns per block, blocks of columns
    const double2 *roots_th, *roots_f1, *mult1;
    const double* dec2;
    const int* colp2;
};

// H -> U: dir_th, dir: exponent signs of the two transforms
__global__ void __launch_bounds__(kMaxThreads)
cols_fwd_kernel(const __grid_constant__ Cols g, const double2* __restrict__ H, double2* __restrict__ U,
                double dir_th, double dir) {
    extern __shared__ __align__(16) unsigned char cols_smem[];
    const int n1 = g.th.n, nf1 = g.f1.n, b = blockIdx.y;
    double2* ub = U + (int64_t)g.nrows * g.nf2 * b;
    if ((int)blockIdx.x >= g.nblocks) {
        // the fine columns without a mode column: a row of them per block of zeros
        const int r = (int)blockIdx.x - g.nblocks;
        for (int p = g.gap_lo + threadIdx.x; p < g.gap_hi; p += blockDim.x)
            ub[(int64_t)r * g.nf2 + p] = make_double2(0.0, 0.0);
        return;
    }
    const int c0 = blockIdx.x * g.C, C = min(g.C, g.ncols - c0);
    double2* A = reinterpret_cast<double2*>(cols_smem);
    double2* B = A + (int64_t)g.C * nf1;
    const double2* hb = H + ((int64_t)b * g.ncols + c0) * n1;
    for (int i = threadIdx.x; i < C * n1; i += blockDim.x) A[i] = hb[i];
    __syncthreads();
    double2* x = fft(A, B, g.th, C, dir_th, g.roots_th);
    double2* y = x == A ? B : A;
    const int pos = (n1 + 1) / 2, neg = n1 / 2;
    for (int c = 0; c < C; ++c) {
        const double d2 = g.dec2[c0 + c];
        for (int p = threadIdx.x; p < nf1; p += blockDim.x) {
            int i = -1;
            if (p < pos) i = p;
            else if (p >= nf1 - neg) i = n1 + (p - nf1);
            double2 v = make_double2(0.0, 0.0);
            if (i >= 0) {
                const double2 a = x[c * n1 + i], f = g.mult1[i];
                v.x = (a.x * f.x - a.y * f.y) * d2;
                v.y = (a.x * f.y + a.y * f.x) * d2;
            }
            y[c * nf1 + p] = v;
        }
    }
    __syncthreads();
    x = fft(y, x, g.f1, C, dir, g.roots_f1);
    // kept rows, the block's columns side by side
    int row0 = g.row0 % nf1;
    if (row0 < 0) row0 += nf1;
    for (int i = threadIdx.x; i < C * g.nrows; i += blockDim.x) {
        const int r = i / C, c = i - r * C;
        int p = row0 + r;
        if (p >= nf1) p -= nf1;
        ub[(int64_t)r * g.nf2 + g.colp2[c0 + c]] = x[c * nf1 + p];
    }
}

// U -> H, the transpose
__global__ void __launch_bounds__(kMaxThreads)
cols_adj_kernel(const __grid_constant__ Cols g, const double2* __restrict__ U, double2* __restrict__ H,
                double dir_th, double dir) {
    extern __shared__ __align__(16) unsigned char cols_smem[];
    const int n1 = g.th.n, nf1 = g.f1.n, b = blockIdx.y;
    const double2* ub = U + (int64_t)g.nrows * g.nf2 * b;
    const int c0 = blockIdx.x * g.C, C = min(g.C, g.ncols - c0);
    double2* A = reinterpret_cast<double2*>(cols_smem);
    double2* B = A + (int64_t)g.C * nf1;
    int row0 = g.row0 % nf1;
    if (row0 < 0) row0 += nf1;
    for (int i = threadIdx.x; i < C * nf1; i += blockDim.x) {
        const int r = i / C, c = i - r * C;
        int p = row0 + r;
        if (p >= nf1) p -= nf1;
        A[c * nf1 + p] = r < g.nrows ? ub[(int64_t)r * g.nf2 + g.colp2[c0 + c]] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    double2* x = fft(A, B, g.f1, C, dir, g.roots_f1);
    double2* y = x == A ? B : A;
    for (int c = 0; c < C; ++c) {
        const double d2 = g.dec2[c0 + c];
        for (int i = threadIdx.x; i < n1; i += blockDim.x) {
            const int k = i < (n1 + 1) / 2 ? i : i - n1;
            const double2 a = x[c * nf1 + (k >= 0 ? k : nf1 + k)], f = g.mult1[i];  // conj(f)
            y[c * n1 + i] = make_double2((a.x * f.x + a.y * f.y) * d2, (a.y * f.x - a.x * f.y) * d2);
        }
    }
    __syncthreads();
    x = fft(y, x, g.th, C, dir_th, g.roots_th);
    double2* hb = H + ((int64_t)b * g.ncols + c0) * n1;
    for (int i = threadIdx.x; i < C * n1; i += blockDim.x) hb[i] = x[i];
}

Div make_div(int d) { return Div{(unsigned)d, d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u}; }

// passes of a 2, 3, 5, 7-smooth length; false for others
bool make_fft(int n, Fft& f) {
    int e2 = 0, e3 = 0, m = n;
    std::vector<int> r;
    for (; m % 2 == 0; m /= 2) ++e2;
    for (; m % 3 == 0; m /= 3) ++e3;
    for (int p : {5, 7})
        for (; m % p == 0; m /= p) r.push_back(p);
    if (m != 1) return false;
    for (; e3 >= 2; e3 -= 2) r.push_back(9);
    if (e3) r.push_back(3);
    while (e2 > 4 || e2 == 3) {
        r.push_back(8);
        e2 -= 3;
    }
    if (e2 == 4) r.push_back(4);
    if (e2 == 4 || e2 == 2) r.push_back(4);
    else if (e2 == 1) r.push_back(2);
    if (r.size() > 12) return false;
    f.n = n;
    f.npass = (int)r.size();
    int ns = 1;
    for (int p = 0; p < f.npass; ++p) {
        f.radix[p] = r[p];
        f.per[p] = make_div(n / r[p]);
        f.ns[p] = make_div(ns);
        ns *= r[p];
    }
    return true;
}

int upload_roots(int n, DevBuf& d, cudaStream_t s) {
    std::vector<double2> w(n);
    for (int k = 0; k < n; ++k) {
        const long double a = 2.0L * 3.14159265358979323846264338327950288L * k / n;
        w[k] = make_double2((double)std::cos(a), (double)std::sin(a));
    }
    PF_TRY(d.alloc(sizeof(double2) * n));
    PF_CUDA(cudaMemcpyAsync(d.p, w.data(), sizeof(double2) * n, cudaMemcpyHostToDevice, s));
    PF_CUDA(cudaStreamSynchronize(s));
    return 0;
}

// threads: about one radix-8 butterfly each (256 threads for the 40 butterflies of one 320-long column
// took 27 us at 0.46 million cells, 64 threads 16; 352 for 324 butterflies 131 us at 3.6 million, 256 94)
int block_threads(int C, int nf1) { return std::min(kMaxThreads, std::max(64, (C * nf1 / 8 + 31) / 32 * 32)); }

// columns per block: those that leave the busiest multiprocessor the fewest columns
int cols_per_block(const NufftGrid& g, int B) {
    int best = 0;
    int64_t least = 0;
    for (int C = 1; C <= 8; ++C) {
        const size_t smem = 2 * sizeof(double2) * (size_t)C * g.nf1;
        if (smem > kMaxSmem) break;
        const int occ = std::min((int)(227 * 1024 / (smem + 1024)), 64 * 1024 / (90 * block_threads(C, g.nf1)));
        const int64_t blocks = (int64_t)((g.ncols + C - 1) / C) * B;
        const int64_t waves = (blocks + (int64_t)148 * occ - 1) / ((int64_t)148 * occ);
        const int64_t cost = C * (waves == 1 ? (blocks + 147) / 148 : waves * occ);
        if (best == 0 || cost < least) {
            best = C;
            least = cost;
        }
    }
    return best;
}

int fill_cols(const NufftGrid& g, const NufftDev& d, int B, Cols& c) {
    make_fft(g.n1, c.th);
    make_fft(g.nf1, c.f1);
    c.ncols = g.ncols;
    c.row0 = g.row0;
    c.nrows = g.nrows;
    c.nf2 = g.nf2;
    c.gap_lo = g.gap_lo;
    c.gap_hi = g.gap_hi;
    c.C = cols_per_block(g, B);
    c.nblocks = (g.ncols + c.C - 1) / c.C;
    c.roots_th = d.roots_th.as<double2>();
    c.roots_f1 = d.roots_f1.as<double2>();
    c.mult1 = d.mult1.as<double2>();
    c.dec2 = d.dec2.as<double>();
    c.colp2 = d.colp2.as<int>();
    return (int)(2 * sizeof(double2) * (size_t)c.C * g.nf1);
}

}  // namespace

int setup_cols(NufftGrid& g, NufftDev& d, int B, cudaStream_t s) {
    Fft th, f1;
    g.cols = 0;
    if (g.fp32 || !g.gap_ok || g.row_wrap || cols_per_block(g, B) < 1 || !make_fft(g.n1, th) || !make_fft(g.nf1, f1) ||
        g.nf1 < g.n1 || (int64_t)g.nf1 * 8 > 65535 || (int64_t)g.nf1 * g.ncols > kColsMostCells)
        return 0;
    // the limit belongs to the kernels, not to a plan: it is the same for every plan and set before any
    // launch, since a plan that set its own size before a launch could lower it under another thread's
    PF_CUDA(cudaFuncSetAttribute(cols_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    PF_CUDA(cudaFuncSetAttribute(cols_adj_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    PF_TRY(upload_roots(g.n1, d.roots_th, s));
    PF_TRY(upload_roots(g.nf1, d.roots_f1, s));
    g.cols = 1;
    return 0;
}

int cols_forward(const NufftGrid& g, NufftDev& d, const double2* H, int B, int iflag, cudaStream_t s) {
    Cols c;
    const int smem = fill_cols(g, d, B, c);
    const int zeros = g.gap_hi > g.gap_lo ? g.nrows : 0;
    cols_fwd_kernel<<<dim3(c.nblocks + zeros, B), block_threads(c.C, c.f1.n), smem, s>>>(c, H, d.U.as<double2>(), -1.0,
                                                                       iflag > 0 ? 1.0 : -1.0);
    return check_launch("cols_fwd_kernel");
}

int cols_adjoint(const NufftGrid& g, NufftDev& d, double2* H, int B, int iflag, cudaStream_t s) {
    Cols c;
    const int smem = fill_cols(g, d, B, c);
    cols_adj_kernel<<<dim3(c.nblocks, B), block_threads(c.C, c.f1.n), smem, s>>>(c, d.U.as<double2>(), H, 1.0, iflag > 0 ? 1.0 : -1.0);
    return check_launch("cols_adj_kernel");
}

}  // namespace pf
