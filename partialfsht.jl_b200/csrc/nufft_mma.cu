// FP64 interpolation and spreading of the NUFFT on the double-precision matrix instruction
// (mma.m8n8k4.f64; the 5th-generation tensor path has no FP64 kind). On sm_100a that instruction
// runs at the FP64 FMA rate (measured: 16.0 cycles per multiprocessor quarter for its 256
// multiply-adds, 2.0 for the 32 of a DFMA), so it adds no peak; what it takes away is everything
// around the multiply-adds. A point's w x w taps are a product of its row and column weights, and
// neighbouring points share fine-grid cells, so
//   type 2:  T[p, r] = sum_c k2[p, c] U[r, c]   (points x columns times columns x rows),
//            f[p]    = sum_r k1[p, r] T[p, r]
//   type 1:  U[c, r] += sum_p k2[p, c] (v[p] k1[p, r])
// with 8 points per product in type 2 and 4 in type 1, whose weights are zero off their windows.
//
// Order of the points. The grid is cut into blocks of columns (CT - w + 1 origin columns, so a
// block's windows span CT = 16 or 24 columns) and each block into strips of four origin rows; the
// points are sorted by block, strip, origin column and laid out in groups of 8 slots, the points
// of a group lying in at most two neighbouring strips of one block (the last slots of a group may
// be empty). A warp takes an item: a stretch of consecutive groups of one block. It walks the
// strips upwards with a window of NT + 1 sets of four rows in registers (the rows that the points
// of two neighbouring strips reach): type 2 loads each next set one strip ahead, type 1 adds each
// set that is left behind to U, so no tile is staged in shared memory and the length of an
// item is free. A group takes NT sets, or all NT + 1 when it reaches into a second strip.
//
// Registers of lane l, t = l % 4, q = l / 4:
//   type 2 (operand B, k = column, n = row and component): win[n][ks] is component q % 2 of row
//           4 n + q / 2 of the window, column 4 ks + t;
//   type 1 (accumulator, m = column, n = row and component): acc[n][i] is both components of row
//           4 n + t of the window, column 8 i + q.
//
// Each batch of 32 slots is staged in shared memory, a lane evaluating one point's weights. The
// weights of a point lie in a row with zeros on both sides (a row's trailing zeros are the next
// one's leading zeros), so a lane reads the weight of any column or row of the window, in or off
// the point's own, at a constant offset from the point's place. The rows are dealt so that the
// stores of 16 lanes and the reads of 4 neighbouring points fall in distinct banks. What these
// kernels are bound by is the instructions around the products (with each product replaced by one
// multiply-add they ran 84-92% of the time at lmax 2048), so everything that depends on the
// points' positions alone is packed into one word per slot at plan time.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.cuh"
#include "nufft_dev.cuh"

namespace pf {

namespace {

constexpr int kWarps = 4;  // items (warps) per block

// columns of the window for kernel width w
__host__ __device__ constexpr int tile_cols(int w) { return w <= 13 ? 16 : 24; }

// x with x s = 1 (mod 16), s odd
__host__ __device__ constexpr int inv16(int s) {
    for (int x = 1; x < 16; x += 2)
        if ((x * s) % 16 == 1) return x;
    return 1;
}

template <int W>
struct Shape {
    static constexpr int CT = tile_cols(W);
    static constexpr int KS = CT / 4;       // column steps of a type-2 product
    static constexpr int MT = CT / 8;       // column tiles of a type-1 product
    static constexpr int NT = (W + 6) / 4;  // row groups that the points of one strip reach
    static constexpr int NW = NT + 1;       // row groups of the window
    // column weights: zeros for the columns -(CT - W) .. CT - 1 of the block around the W
    static constexpr int F2 = CT - W, S2 = CT | 1;
    // row weights: the point's origin row is row 0 .. 7 of the window
    static constexpr int F1 = 7, P1 = 4 * NW - W > F1 ? 4 * NW - W : F1, S1 = (W + P1) | 1;
};

template <int W>
struct Stage {
    static constexpr int N1 = Shape<W>::F1 + 32 * Shape<W>::S1;
    static constexpr int N2 = Shape<W>::F2 + 32 * Shape<W>::S2;
    double k[N1 + N2];  // row weights, then column weights
};
template <int W>
struct SpreadStage : Stage<W> {
    double2 v[32];  // the points' values
};

// A slot's word: where in Stage::k the group's window's row 0 (bits 0-11) and the block's column 0
// (bits 12-23) find the point's weights, the strips that the window moves up before the slot's
// group (24-30), and whether the group reaches into a second strip (31).
constexpr int kMaxAdvance = 127;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// the first product of a sum
__device__ __forceinline__ void dmma0(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};"
                 : "=d"(c[0]), "=d"(c[1])
                 : "d"(a), "d"(b), "d"(0.0));
}

// row of lane l's point: a permutation of 0 .. 31 with S x row = 4 (l % 4) + (l / 4) % 4 (mod 16)
template <int S>
__device__ __forceinline__ int stage_row(int l) {
    return (l & 16) | (((((l & 3) << 2) | ((l >> 2) & 3)) * inv16(S)) & 15);
}

template <int W>
__device__ __forceinline__ void clear_stage(Stage<W>& st, int lane) {
    for (int i = lane; i < Stage<W>::N1 + Stage<W>::N2; i += 32) st.k[i] = 0.0;
}

// The tap weights' coefficients in shared memory, (even, odd) pairs by power of v^2 for each
// mirrored pair of taps (and the middle tap of an odd width): a lane evaluates its row and
// column weights from the same loads. (As operands from the constant bank they cost two register
// moves each: 400 of the 1120 warp instructions per batch of 32 points at w = 9.)
template <int W>
struct Coef {
    static constexpr int NC = EsHorner<W>::NC;
    static constexpr int N2 = (NC + 1) / 2;
    double2 c[(W + 1) / 2][N2];
};

template <int W>
__device__ __forceinline__ void load_coef(Coef<W>& cf) {
    using C = Coef<W>;
    const double* src = EsHorner<W>::coef();
    for (int i = threadIdx.x; i < (W + 1) / 2 * C::N2; i += blockDim.x) {
        const int a = i / C::N2, k = 2 * (i % C::N2);
        cf.c[a][k / 2] = make_double2(src[a * C::NC + k], k + 1 < C::NC ? src[a * C::NC + k + 1] : 0.0);
    }
}

// i modulo n for -n <= i < 2 n
__device__ __forceinline__ int wrap_once(int i, int n) { return i < 0 ? i + n : i >= n ? i - n : i; }

// plan time: the slots of the groups (of 8 slots; items start at multiples of 32 slots)
template <int W>
__global__ void mma_slots_kernel(const double2* __restrict__ g, const int* __restrict__ sidx,
                                 const MmaGroup* __restrict__ groups, int64_t nslots, int nrows, int nf2,
                                 int row_wrap, double2* __restrict__ off, int2* __restrict__ meta) {
    using H = Shape<W>;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nslots) return;  // whole warps: nslots is a multiple of 32
    const MmaGroup r = groups[i >> 3];
    const int k = (int)(i & 7), lane = (int)(i & 31);
    double2 v = make_double2(0.0, 0.0);
    int c0 = 0, row = 0, place = -1;
    if (k < r.n) {
        place = sidx[r.first + k];
        const double2 p = g[place];
        const int i10 = (int)ceil(p.x - 0.5 * W), i20 = (int)ceil(p.y - 0.5 * W);
        v.x = ((double)i10 - p.x) + (0.5 * W - 0.5);
        v.y = ((double)i20 - p.y) + (0.5 * W - 0.5);
        // the sort put every origin into its block and into the group's strips
        c0 = min(max(wrap_once(i20, nf2) - r.col, 0), H::CT - W);
        row = min(max((row_wrap ? wrap_once(i10, nrows) : i10) - 4 * r.strip, 0), 7);
    }
    const unsigned second = (__ballot_sync(0xffffffffu, row >= 4) >> (lane & 24)) & 0xff ? 1u : 0u;
    const unsigned a1 = H::F1 + stage_row<H::S1>(lane) * H::S1 - row;
    const unsigned a2 = Stage<W>::N1 + H::F2 + stage_row<H::S2>(lane) * H::S2 - c0;
    off[i] = v;
    meta[i] = make_int2((int)(a1 | (a2 << 12) | ((unsigned)r.advance << 24) | (second << 31)), place);
}

// this lane's point's weights. The mirrored taps a and W - 1 - a come from one even and one odd
// Horner chain, p_a(v) = E(v^2) + v O(v^2), as in es_pair.
// w1, w2: the shared addresses of its rows
__device__ __forceinline__ void put(unsigned a, double x) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}
template <int W>
__device__ __forceinline__ void stage_weights(unsigned w1, unsigned w2, const Coef<W>& cf, double2 v) {
    const double u1 = v.x * v.x, u2 = v.y * v.y;
    constexpr int N2 = Coef<W>::N2;
#pragma unroll
    for (int a = 0; a < (W + 1) / 2; ++a) {
        const bool mid = 2 * a == W - 1;
        double2 c = cf.c[a][N2 - 1];
        double e1 = c.x, o1 = c.y, e2 = c.x, o2 = c.y;
#pragma unroll
        for (int i = N2 - 2; i >= 0; --i) {
            c = cf.c[a][i];
            e1 = fma(e1, u1, c.x);
            e2 = fma(e2, u2, c.x);
            if (!mid) {
                o1 = fma(o1, u1, c.y);
                o2 = fma(o2, u2, c.y);
            }
        }
        put(w1 + 8 * a, mid ? e1 : fma(v.x, o1, e1));
        put(w2 + 8 * a, mid ? e2 : fma(v.y, o2, e2));
        if (!mid) {
            put(w1 + 8 * (W - 1 - a), fma(-v.x, o1, e1));
            put(w2 + 8 * (W - 1 - a), fma(-v.y, o2, e2));
        }
    }
}

// the double at shared address a
__device__ __forceinline__ double weight(unsigned a) {
    double x;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a) : "memory");
    return x;
}

template <int W>
__global__ void __launch_bounds__(kWarps * 32, W <= 13 ? 5 : 3)
interp_mma_kernel(const double2* __restrict__ off, const int2* __restrict__ meta,
                  const int4* __restrict__ items, int nitems, const double2* __restrict__ U,
                  int nrows, int nf2, int row_wrap, int64_t M, double2* __restrict__ f) {
    using H = Shape<W>;
    extern __shared__ __align__(16) unsigned char mma_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.x * kWarps + warp;
    __shared__ Coef<W> cf;
    load_coef<W>(cf);
    __syncthreads();
    if (slot >= nitems) return;
    const int4 it = items[slot];  // first origin row and column, slots [z, w)
    // the transform
    U += (int64_t)nrows * nf2 * blockIdx.y;
    f += M * blockIdx.y;
    const unsigned never = (unsigned)nrows >> 31;  // 0, which the compiler does not know
    Stage<W>& st = reinterpret_cast<Stage<W>*>(mma_smem)[warp];
    const int t = lane & 3;
    const double2* po = off + it.z + lane;
    const int2* pm = meta + it.z + lane;
    // each batch's slots load under the batch before
    double2 v = *po;
    int2 m = *pm;
    int col[H::KS];
#pragma unroll
    for (int ks = 0; ks < H::KS; ++ks) col[ks] = 2 * wrap(it.y + 4 * ks + t, nf2) + ((lane >> 2) & 1);
    int top = it.x + (lane >> 3);  // this lane's row of the window's first set
    auto load = [&](double (&w)[H::KS], int set) {
        int gr = top + 4 * set;
        if (row_wrap) gr = wrap(gr, nrows);
        const double* row = reinterpret_cast<const double*>(U) + 2 * (int64_t)gr * nf2;
        const bool ok = gr >= 0 && gr < nrows;
#pragma unroll
        for (int ks = 0; ks < H::KS; ++ks) w[ks] = ok ? row[col[ks]] : 0.0;
    };
    double win[H::NW][H::KS];
#pragma unroll
    for (int n = 0; n < H::NW; ++n) load(win[n], n);
    clear_stage<W>(st, lane);
    unsigned w1 = (unsigned)__cvta_generic_to_shared(st.k) + 8 * (H::F1 + stage_row<H::S1>(lane) * H::S1);
    unsigned w2 = (unsigned)__cvta_generic_to_shared(st.k) + 8 * (Stage<W>::N1 + H::F2 + stage_row<H::S2>(lane) * H::S2);
    asm volatile("" : "+r"(w1), "+r"(w2));  // kept in registers, not worked out anew for each batch
    const unsigned k0 = (unsigned)__cvta_generic_to_shared(st.k) + 8 * t;
    // operands that sum a column of lanes t into the lane t = 0: real parts into column 0 of the
    // product, imaginary parts into column 1
    const double one0 = lane < 4 ? 1.0 : 0.0, one1 = lane >= 4 && lane < 8 ? 1.0 : 0.0;
    for (int left = it.w - it.z; left > 0; left -= 32) {
        __syncwarp();
        stage_weights<W>(w1, w2, cf, v);
        const int2 mc = m;
        const unsigned used = __ballot_sync(0xffffffffu, m.y >= 0);
        if (left > 32) {
            po += 32;
            pm += 32;
            v = *po;
            m = *pm;
        }
        __syncwarp();
#pragma unroll 1
        for (int k = lane >> 2; k < 32; k += 8) {
            if (!((used >> (k & 24)) & 0xff)) break;  // only the item's last groups are empty
            const unsigned x = (unsigned)__shfl_sync(0xffffffffu, mc.x, k);
            unsigned adv = (x >> 24) & kMaxAdvance;
            if (adv) {
                // move the window up to the group's strip
                if (adv >= H::NW) {
                    top += 4 * adv;
#pragma unroll
                    for (int n = 0; n < H::NW; ++n) load(win[n], n);
                    adv = 0;
                }
#pragma unroll 1
                for (; adv; --adv) {
#pragma unroll
                    for (int ks = 0; ks < H::KS; ++ks)
#pragma unroll
                        for (int n = 0; n + 1 < H::NW; ++n) win[n][ks] = win[n + 1][ks];
                    // the new last set is read by a group of two strips or, at the earliest, in
                    // the next strip, so its loads are covered by this strip's products
                    top += 4;
                    load(win[H::NW - 1], H::NW - 1);
                }
            }
            const unsigned a1 = k0 + ((x & 0xfff) << 3), a2 = k0 + ((x >> 9) & 0x7ff8);
            double a[H::KS];
#pragma unroll
            for (int ks = 0; ks < H::KS; ++ks) a[ks] = weight(a2 + 32 * ks);
            double k1[H::NT];
#pragma unroll
            for (int n = 0; n < H::NT; ++n) k1[n] = weight(a1 + 32 * n);
            double c[H::NT][2];
#pragma unroll
            for (int n = 0; n < H::NT; ++n) dmma0(c[n], a[0], win[n][0]);
#pragma unroll
            for (int ks = 1; ks < H::KS; ++ks)
#pragma unroll
                for (int n = 0; n < H::NT; ++n) dmma(c[n], a[ks], win[n][ks]);
            double2 sum = make_double2(c[0][0] * k1[0], c[0][1] * k1[0]);
#pragma unroll
            for (int n = 1; n < H::NT; ++n) {
                sum.x = fma(c[n][0], k1[n], sum.x);
                sum.y = fma(c[n][1], k1[n], sum.y);
            }
            // a loop, so that the products are branched around and not predicated
#pragma unroll 1
            for (unsigned z = x >> 31; z != 0; z = never) {
                constexpr int n = H::NT;
                const double kl = weight(a1 + 32 * n);
                double d[2];
                dmma0(d, a[0], win[n][0]);
#pragma unroll
                for (int ks = 1; ks < H::KS; ++ks) dmma(d, a[ks], win[n][ks]);
                sum.x = fma(d[0], kl, sum.x);
                sum.y = fma(d[1], kl, sum.y);
            }
            double r[2];
            dmma0(r, sum.x, one0);
            dmma(r, sum.y, one1);
            const int p = __shfl_sync(0xffffffffu, mc.y, k);
            if (t == 0 && p >= 0) f[p] = make_double2(r[0], r[1]);
        }
    }
}

template <int W>
__global__ void __launch_bounds__(kWarps * 32, W <= 9 ? 5 : W <= 13 ? 4 : 3)
spread_mma_kernel(const double2* __restrict__ off, const int2* __restrict__ meta,
                  const int4* __restrict__ items, int nitems, const double2* __restrict__ fin,
                  int nrows, int nf2, int row_wrap, int64_t M, double2* __restrict__ U) {
    using H = Shape<W>;
    extern __shared__ __align__(16) unsigned char mma_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.x * kWarps + warp;
    __shared__ Coef<W> cf;
    load_coef<W>(cf);
    __syncthreads();
    if (slot >= nitems) return;
    const int4 it = items[slot];  // first origin row and column, slots [z, w)
    // the transform
    U += (int64_t)nrows * nf2 * blockIdx.y;
    fin += M * blockIdx.y;
    const unsigned never = (unsigned)nrows >> 31;  // 0, which the compiler does not know
    SpreadStage<W>& st = reinterpret_cast<SpreadStage<W>*>(mma_smem)[warp];
    const int t = lane & 3, q = lane >> 2;
    const double2* po = off + it.z + lane;
    const int2* pm = meta + it.z + lane;
    // each batch's slots and values load while the batch before is added; empty slots add 0
    auto value = [&](int j) { return j >= 0 ? fin[j] : make_double2(0.0, 0.0); };
    double2 v = *po;
    int2 m = *pm;
    double2 fv = value(m.y);
    int col[H::MT];
#pragma unroll
    for (int i = 0; i < H::MT; ++i) col[i] = wrap(it.y + 8 * i + q, nf2);
    double acc[H::NW][H::MT][2];
#pragma unroll
    for (int n = 0; n < H::NW; ++n)
#pragma unroll
        for (int i = 0; i < H::MT; ++i) acc[n][i][0] = acc[n][i][1] = 0.0;
    int top = it.x + t;  // this lane's row of the window's first set
    // add one set of rows to U (neighbouring items' windows overlap it)
    auto flush = [&](const double (&w)[H::MT][2], int set) {
        int gr = top + 4 * set;
        if (row_wrap) gr = wrap(gr, nrows);
        if (gr < 0 || gr >= nrows) return;
#pragma unroll
        for (int i = 0; i < H::MT; ++i) {
            if (w[i][0] != 0.0 || w[i][1] != 0.0) {
                double* d = reinterpret_cast<double*>(U + (int64_t)gr * nf2 + col[i]);
                atomicAdd(d, w[i][0]);
                atomicAdd(d + 1, w[i][1]);
            }
        }
    };
    clear_stage<W>(st, lane);
    unsigned w1 = (unsigned)__cvta_generic_to_shared(st.k) + 8 * (H::F1 + stage_row<H::S1>(lane) * H::S1);
    unsigned w2 = (unsigned)__cvta_generic_to_shared(st.k) + 8 * (Stage<W>::N1 + H::F2 + stage_row<H::S2>(lane) * H::S2);
    asm volatile("" : "+r"(w1), "+r"(w2));  // kept in registers, not worked out anew for each batch
    const unsigned kr = (unsigned)__cvta_generic_to_shared(st.k) + 8 * (q >> 1);
    const unsigned kc = (unsigned)__cvta_generic_to_shared(st.k) + 8 * q;
    const unsigned kv = (unsigned)__cvta_generic_to_shared(st.v) + 16 * t + 8 * (q & 1);
    for (int left = it.w - it.z; left > 0; left -= 32) {
        __syncwarp();
        stage_weights<W>(w1, w2, cf, v);
        st.v[lane] = fv;
        const int mc = m.x;
        const unsigned used = __ballot_sync(0xffffffffu, m.y >= 0);
        if (left > 32) {
            po += 32;
            pm += 32;
            v = *po;
            m = *pm;
        }
        __syncwarp();
        fv = value(left > 32 ? m.y : -1);
#pragma unroll 1
        for (int k = 0; k < 32; k += 4) {
            if (!((used >> k) & 15)) continue;  // an empty half of a group
            const unsigned x = (unsigned)__shfl_sync(0xffffffffu, mc, k + t);
            unsigned adv = (k & 4) ? 0 : (x >> 24) & kMaxAdvance;
            if (adv) {
                // move the window up to the group's strip; what is left behind is complete
                const int n_out = min(adv, (unsigned)H::NW);
#pragma unroll 1
                for (int n = 0; n < n_out; ++n) {
                    flush(acc[0], n);
#pragma unroll
                    for (int i = 0; i < H::MT; ++i)
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
#pragma unroll
                            for (int s = 0; s + 1 < H::NW; ++s) acc[s][i][y] = acc[s + 1][i][y];
                            acc[H::NW - 1][i][y] = 0.0;
                        }
                }
                top += 4 * adv;
            }
            const unsigned a1 = kr + ((x & 0xfff) << 3), a2 = kc + ((x >> 9) & 0x7ff8);
            const double val = weight(kv + 16 * k);
            double a[H::MT], b[H::NT];
#pragma unroll
            for (int i = 0; i < H::MT; ++i) a[i] = weight(a2 + 64 * i);
#pragma unroll
            for (int n = 0; n < H::NT; ++n) b[n] = val * weight(a1 + 32 * n);
#pragma unroll
            for (int n = 0; n < H::NT; ++n)
#pragma unroll
                for (int i = 0; i < H::MT; ++i) dmma(acc[n][i], a[i], b[n]);
            // a loop, so that the products are branched around and not predicated
#pragma unroll 1
            for (unsigned z = x >> 31; z != 0; z = never) {
                const double bl = val * weight(a1 + 32 * H::NT);
#pragma unroll
                for (int i = 0; i < H::MT; ++i) dmma(acc[H::NT][i], a[i], bl);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < H::NW; ++n) flush(acc[n], n);
}

template <class K>
int set_smem(K kernel, size_t bytes) {
    if (bytes > 40 * 1024)  // (a block has some static shared memory too)
        PF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return 0;
}

template <int W>
int launch_interp_mma(const NufftGrid& g, NufftDev& d, double2* f, int B, cudaStream_t s) {
    if constexpr (W < kMmaInterpWidth) {
        set_error("interpolation of this width does not run on the matrix instruction");
        return 7;
    } else {
        const size_t smem = kWarps * sizeof(Stage<W>);
        PF_TRY(set_smem(interp_mma_kernel<W>, smem));
        interp_mma_kernel<W><<<dim3((g.nitems + kWarps - 1) / kWarps, B), kWarps * 32, smem, s>>>(
            d.soff.as<double2>(), d.smeta.as<int2>(), d.items.as<int4>(), g.nitems, d.U.as<double2>(), g.nrows, g.nf2,
            g.row_wrap, g.M, f);
        return check_launch("interp_mma_kernel");
    }
}

template <int W>
int launch_spread_mma(const NufftGrid& g, NufftDev& d, const double2* f, int B, cudaStream_t s) {
    const size_t smem = kWarps * sizeof(SpreadStage<W>);
    PF_TRY(set_smem(spread_mma_kernel<W>, smem));
    spread_mma_kernel<W><<<dim3((g.nitems + kWarps - 1) / kWarps, B), kWarps * 32, smem, s>>>(
        d.soff.as<double2>(), d.smeta.as<int2>(), d.items.as<int4>(), g.nitems, f, g.nrows, g.nf2, g.row_wrap, g.M,
        d.U.as<double2>());
    return check_launch("spread_mma_kernel");
}

template <int W>
int launch_mma_slots(const NufftGrid& g, NufftDev& d, const double2* gg, const int* sidx,
                     const MmaGroup* groups, int64_t nslots, cudaStream_t s) {
    mma_slots_kernel<W><<<(unsigned)((nslots + 255) / 256), 256, 0, s>>>(
        gg, sidx, groups, nslots, g.nrows, g.nf2, g.row_wrap, d.soff.as<double2>(), d.smeta.as<int2>());
    return check_launch("mma_slots_kernel");
}

#define PF_MMA_WIDTHS(CALL)                                                                    \
    switch (g.w) {                                                                             \
        case 2: return CALL(2); case 3: return CALL(3); case 4: return CALL(4);                \
        case 5: return CALL(5); case 6: return CALL(6); case 7: return CALL(7);                \
        case 8: return CALL(8); case 9: return CALL(9); case 10: return CALL(10);              \
        case 11: return CALL(11); case 12: return CALL(12); case 13: return CALL(13);          \
        case 14: return CALL(14); case 15: return CALL(15); case 16: return CALL(16);          \
        default: break;                                                                        \
    }                                                                                          \
    set_error("unsupported NUFFT kernel width");                                               \
    return 7;

}  // namespace

int mma_tile_cols(int w) { return tile_cols(w); }

int mma_max_advance() { return kMaxAdvance; }

int mma_fill_slots(const NufftGrid& g, NufftDev& d, const double2* gg, const int* sidx,
                   const MmaGroup* groups, int64_t nslots, cudaStream_t s) {
    if (nslots == 0) return 0;
#define PF_CALL(W) launch_mma_slots<W>(g, d, gg, sidx, groups, nslots, s)
    PF_MMA_WIDTHS(PF_CALL)
#undef PF_CALL
}

int interp_mma(const NufftGrid& g, NufftDev& d, double2* f, int B, cudaStream_t s) {
    if (g.nitems == 0) return 0;
#define PF_CALL(W) launch_interp_mma<W>(g, d, f, B, s)
    PF_MMA_WIDTHS(PF_CALL)
#undef PF_CALL
}

int spread_mma(const NufftGrid& g, NufftDev& d, const double2* f, int B, cudaStream_t s) {
    if (g.nitems == 0) return 0;
#define PF_CALL(W) launch_spread_mma<W>(g, d, f, B, s)
    PF_MMA_WIDTHS(PF_CALL)
#undef PF_CALL
}

}  // namespace pf
