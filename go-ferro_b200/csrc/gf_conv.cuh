// Magnetostatic convolution H = -F^-1[ N_k . F[M] ] / (dx dy dz) of a stage
// in three launches of the engine's own FFTs (FP64 and FP32), for grids whose
// sides have the factors 2, 3, 5 and whose planes fit in shared memory.
//
//   k_conv_fwd  one block per x-plane and component: M (Ms m formed on the
//               fly), real transform along z of row pairs packed as one
//               complex row, complex transform along y, the half spectrum of
//               the plane to memory.
//   k_conv_x    one block per group of (k_y, k_z) columns, all three
//               components: transform along x, the tensor product, inverse
//               transform along x, in place.  FP64 takes the reference's nine
//               complex spectra as they are (k_demag_mul); FP32 the six real
//               ones of the symmetric tensor (k_demag_mul_f32).
//   k_conv_inv  the inverse of k_conv_fwd, writing H.
//
// cuFFT's batched 3-D pair plus the source and product kernels are eight to
// twelve launches that each pass over the spectrum; here it is written and
// read twice and stays in L2 between the launches for films up to ~2 M cells
// in FP32.  Small films are bound by launch latency (three launches instead
// of eight), large ones by the shared-memory passes and the barriers between
// them (256x256x32 FP32: 43 + 50 + 33 us, where its 84 bytes per cell take 27).
//
// The transforms are Stockham autosort passes in shared memory, two buffers
// used in turn, each butterfly in registers.  A pass spreads its butterflies
// over the block with the line index fastest, so that neighbouring threads
// touch neighbouring words; the twiddles sit in shared memory.  A small film
// keeps a warp or two per scheduler busy and is bound by the instructions and
// waits of one thread: the copies between memory and shared memory, the row
// packing and the tensor product are phases of their own that all threads
// share, by cp.async or with four items' loads of a thread in flight (folded
// into the passes next to them, 64x64x16 and 120x90x20 FP64 steps took 0.110
// and 0.238 ms instead of 0.098 and 0.179).  Radices go up to 8: 16
// along x saves a pass but halves the butterflies and needs twice the
// registers (128x128x32 FP64 step 0.309 ms against 0.299, 120x90x20 FP32 0.129
// against 0.124).
// Unnormalised in both directions, as cuFFT is (the tables hold 1/n).
#pragma once

#include "gf_column.cuh"
#include "gf_demag.cuh"

namespace gf {

template <class R> struct cx_of;
template <> struct cx_of<float> { using type = float2; };
template <> struct cx_of<double> { using type = double2; };
template <class R> using Cx = typename cx_of<R>::type;

// Threads of a block and the blocks per SM its registers allow.  A film's
// planes should all be resident at once (a second, nearly empty wave costs a
// whole block time): FP32 planes take 40 registers without a spill, 6 blocks
// (256x256x32: 38 us per k_conv_fwd, 45 with 5 blocks); FP64 80 registers, 3
// blocks (120x90x20 step 0.164 ms, 2 blocks 0.191).  128 threads per plane block: 0.2 to
// 12 % slower steps on small films; 512: 10 to 25 %.
constexpr int kConvThreads = 256;
template <class R> constexpr int kConvPlaneBlocks = sizeof(R) == 4 ? 6 : 3;
template <class R> constexpr int kConvXBlocks = sizeof(R) == 4 ? 4 : 3;
constexpr size_t kConvMaxSmem = 224 * 1024;
constexpr int kConvMaxPass = 8;
constexpr int kConvMaxSide = 2048;

// quotient of 0 <= n < 2^20 by a fixed d (1 <= d < 2^12): umulhi by ceil(2^32 / d)
struct ConvDiv {
    unsigned m, d;
    __host__ __device__ int div(int n) const {
#ifdef __CUDA_ARCH__
        return d == 1u ? n : (int)__umulhi((unsigned)n, m);
#else
        return d == 1u ? n : (int)(((unsigned long long)(unsigned)n * m) >> 32);
#endif
    }
};
inline ConvDiv conv_div(int d) { return ConvDiv{(unsigned)((4294967296ull + (unsigned)d - 1) / (unsigned)d), (unsigned)d}; }

// passes of one transform length
struct ConvLen {
    int n, np;
    int rad[kConvMaxPass];
    int l[kConvMaxPass];          // product of the earlier radices
    ConvDiv dl[kConvMaxPass];
    int tw;                       // offset of this length's table w_n[k] = exp(-2 pi i k / n)
};

struct ConvGeom {
    int nx, ny, nz, nzc;          // nzc = nz / 2 + 1
    long n, nk;                   // cells; half-spectrum points
    int pairs, pitch;             // row pairs of a plane; words per packed row (odd)
    int plane;                    // words of one plane buffer
    ConvLen lx, ly, lz;
    ConvDiv dpairs, dnz, dnzc;
    int cols, g, groups;          // columns of k_conv_x: all, per block, blocks
    ConvDiv dlines, dg;           // by 3 g and by g
};

// twiddles go by cp.async, so that no thread waits for them before its data loads
__device__ __forceinline__ void conv_copy(float2* d, const float2* g) { cp_async8(d, g); }
__device__ __forceinline__ void conv_copy(double2* d, const double2* g) { cp_async16(d, g); }
// n twiddles into shared memory (before the block's next cp_async_wait_all and barrier)
template <class C> __device__ __forceinline__ void conv_twiddles(C* d, const C* g, int n) {
    for (int q = threadIdx.x; q < n; q += blockDim.x) conv_copy(d + q, g + q);
    cp_async_commit();
}
template <class C> __device__ __forceinline__ C cadd_(C a, C b) { return C{a.x + b.x, a.y + b.y}; }
template <class C> __device__ __forceinline__ C csub_(C a, C b) { return C{a.x - b.x, a.y - b.y}; }
template <class C> __device__ __forceinline__ C cmul_(C a, C b) { return C{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
// a times -i (forward) or +i (inverse)
template <bool INV, class C> __device__ __forceinline__ C crot_(C a) { return INV ? C{-a.y, a.x} : C{a.y, -a.x}; }

// cos and sin of 2 pi k / n at compile time: folded into the first octant,
// then the Taylor series (|x| <= pi / 4: 1e-17 after 11 terms)
__host__ __device__ constexpr double conv_series(double x, bool sine) {
    double t = sine ? x : 1., s = t;
    for (int q = 1; q < 12; q++) {
        const double d = sine ? (2. * q) * (2. * q + 1.) : (2. * q - 1.) * (2. * q);
        t = -t * x * x / d;
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double conv_cs(int k, int n, bool sine) {
    // eighths of a turn: a = 8 k / n
    k %= n;
    const int oct = 8 * k / n;                       // 0..7
    const int r = 8 * k - oct * n;                   // remainder in (1/8n) turns
    const bool odd = oct & 1;
    const double x = 2. * kPi * (double)(odd ? n - r : r) / (8. * n);
    const double c = conv_series(x, false), si = conv_series(x, true);
    // angle = oct * pi / 4 + pi / 4 - x (odd) or + x (even)
    switch (oct) {
        case 0: return sine ? si : c;
        case 1: return sine ? c : si;
        case 2: return sine ? c : -si;
        case 3: return sine ? si : -c;
        case 4: return sine ? -si : -c;
        case 5: return sine ? -c : -si;
        case 6: return sine ? -c : si;
        default: return sine ? -si : c;
    }
}

// first factor of a composite radix (8, 6)
__host__ __device__ constexpr int conv_f1(int n) {
    return n > 5 ? 2 : n;
}

template <int RAD, bool INV, class R>
__device__ __forceinline__ void conv_dft(Cx<R> (&v)[RAD]);

// v[N2 n1 + n2] -> X[k1 + N1 k2]: N2 transforms of length N1, twiddles, N1 of length N2
template <int N1, int N2, bool INV, class R, int K1, int Q>
__device__ __forceinline__ void conv_twid(Cx<R>& c) {
    constexpr R wr = R(conv_cs(K1 * Q, N1 * N2, false)), wi = R((INV ? 1. : -1.) * conv_cs(K1 * Q, N1 * N2, true));
    c = Cx<R>{c.x * wr - c.y * wi, c.x * wi + c.y * wr};
}
template <int N1, int N2, bool INV, class R, int Q>
__device__ __forceinline__ void conv_col(Cx<R> (&v)[N1 * N2]) {
    if constexpr (Q < N2) {
        Cx<R> t[N1];
#pragma unroll
        for (int a = 0; a < N1; a++) t[a] = v[N2 * a + Q];
        conv_dft<N1, INV, R>(t);
        if constexpr (Q > 0) {
            static_assert(N1 == 2);
            conv_twid<N1, N2, INV, R, 1, Q>(t[1]);
        }
#pragma unroll
        for (int a = 0; a < N1; a++) v[N2 * a + Q] = t[a];
        conv_col<N1, N2, INV, R, Q + 1>(v);
    }
}

// DFT of RAD points in registers
template <int RAD, bool INV, class R>
__device__ __forceinline__ void conv_dft(Cx<R> (&v)[RAD]) {
    using C = Cx<R>;
    if constexpr (RAD == 2) {
        const C a = v[0];
        v[0] = cadd_(a, v[1]); v[1] = csub_(a, v[1]);
    } else if constexpr (RAD == 3) {
        const R s = R(0.86602540378443864676);
        const C t = cadd_(v[1], v[2]), d = csub_(v[1], v[2]);
        const C m = C{v[0].x - R(0.5) * t.x, v[0].y - R(0.5) * t.y}, r = crot_<INV>(C{s * d.x, s * d.y});
        v[0] = cadd_(v[0], t); v[1] = cadd_(m, r); v[2] = csub_(m, r);
    } else if constexpr (RAD == 4) {
        const C a = cadd_(v[0], v[2]), b = csub_(v[0], v[2]), c = cadd_(v[1], v[3]), d = crot_<INV>(csub_(v[1], v[3]));
        v[0] = cadd_(a, c); v[1] = cadd_(b, d); v[2] = csub_(a, c); v[3] = csub_(b, d);
    } else if constexpr (RAD == 5) {
        const R c1 = R(0.30901699437494742410), c2 = R(-0.80901699437494742410);
        const R s1 = R(0.95105651629515357212), s2 = R(0.58778525229247312917);
        const C t1 = cadd_(v[1], v[4]), t2 = cadd_(v[2], v[3]), d1 = csub_(v[1], v[4]), d2 = csub_(v[2], v[3]);
        const C m1 = C{v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y};
        const C m2 = C{v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y};
        const C r1 = crot_<INV>(C{s1 * d1.x + s2 * d2.x, s1 * d1.y + s2 * d2.y});
        const C r2 = crot_<INV>(C{s2 * d1.x - s1 * d2.x, s2 * d1.y - s1 * d2.y});
        v[0] = cadd_(v[0], cadd_(t1, t2));
        v[1] = cadd_(m1, r1); v[4] = csub_(m1, r1); v[2] = cadd_(m2, r2); v[3] = csub_(m2, r2);
    } else {
        constexpr int N1 = conv_f1(RAD), N2 = RAD / N1;
        conv_col<N1, N2, INV, R, 0>(v);
        C o[RAD];
#pragma unroll
        for (int a = 0; a < N1; a++) {
            C t[N2];
#pragma unroll
            for (int q = 0; q < N2; q++) t[q] = v[N2 * a + q];
            conv_dft<N2, INV, R>(t);
#pragma unroll
            for (int q = 0; q < N2; q++) o[a + N1 * q] = t[q];
        }
#pragma unroll
        for (int q = 0; q < RAD; q++) v[q] = o[q];
    }
}

// pass p of a transform of `lines` lines from x to y: point e of line q at
// e es + q ls (dlines divides by lines)
template <int RAD, bool INV, class R>
__device__ __forceinline__ void conv_pass(const Cx<R>* __restrict__ x, Cx<R>* __restrict__ y, const ConvLen& L, int p, int lines,
                                          ConvDiv dlines, int es, int ls, const Cx<R>* __restrict__ tw) {
    using C = Cx<R>;
    const int m = L.n / RAD, l = L.l[p], step = m / l;
    for (int it = threadIdx.x; it < lines * m; it += blockDim.x) {
        const int j = dlines.div(it), q = it - j * lines;
        const int jl = L.dl[p].div(j), jr = j - jl * l;
        C v[RAD];
        const C* xs = x + j * es + q * ls;
#pragma unroll
        for (int r = 0; r < RAD; r++) v[r] = xs[r * m * es];
        if (l > 1) {
            const int ws = jr * step;
#pragma unroll
            for (int r = 1; r < RAD; r++) {
                C w = tw[r * ws];
                if (INV) w.y = -w.y;
                v[r] = cmul_(v[r], w);
            }
        }
        conv_dft<RAD, INV, R>(v);
        C* ys = y + (jl * l * RAD + jr) * es + q * ls;
#pragma unroll
        for (int r = 0; r < RAD; r++) ys[r * l * es] = v[r];
    }
}

// all passes of a transform; a holds the input, the buffers are used in
// turn, and the result's buffer is returned
template <bool INV, class R>
__device__ __forceinline__ Cx<R>* conv_fft(Cx<R>* a, Cx<R>* b, const ConvLen& L, int lines, ConvDiv dlines, int es, int ls,
                                           const Cx<R>* __restrict__ tw) {
    for (int p = 0; p < L.np; p++) {
        switch (L.rad[p]) {
            case 8: conv_pass<8, INV, R>(a, b, L, p, lines, dlines, es, ls, tw); break;
            case 6: conv_pass<6, INV, R>(a, b, L, p, lines, dlines, es, ls, tw); break;
            case 5: conv_pass<5, INV, R>(a, b, L, p, lines, dlines, es, ls, tw); break;
            case 4: conv_pass<4, INV, R>(a, b, L, p, lines, dlines, es, ls, tw); break;
            case 3: conv_pass<3, INV, R>(a, b, L, p, lines, dlines, es, ls, tw); break;
            default: conv_pass<2, INV, R>(a, b, L, p, lines, dlines, es, ls, tw); break;
        }
        __syncthreads();
        Cx<R>* t = a; a = b; b = t;
    }
    return a;
}

// n items of the block, four loads of a thread in flight
template <class V, class Ld, class St>
__device__ __forceinline__ void conv_items4(int n, Ld load, St store) {
    for (int it0 = threadIdx.x; it0 < n; it0 += 4 * blockDim.x) {
        V v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int it = it0 + u * blockDim.x;
            if (it < n) v[u] = load(it);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int it = it0 + u * blockDim.x;
            if (it < n) store(it, v[u]);
        }
    }
}

// Block (plane i, component c).  mats != null: the input is m and the source
// is Ms m in ferromagnetic cells, 0 elsewhere (k_mag_source); otherwise the
// input is the source itself.
template <class R>
static __global__ void __launch_bounds__(kConvThreads, kConvPlaneBlocks<R>) k_conv_fwd(const __grid_constant__ ConvGeom G, F3T<R> in, const uint8_t* __restrict__ mid,
                                                          const DevMatT<R>* __restrict__ mats, int nmat,
                                                          const Cx<R>* __restrict__ tw_g, Cx<R>* __restrict__ spec) {
    using C = Cx<R>;
    GF_EXTERN_SMEM(unsigned char, smem_raw);
    C* a = reinterpret_cast<C*>(smem_raw);
    C* b = a + G.plane;
    C* tw = b + G.plane;                               // y then z tables
    __shared__ R sMs[kMaxMat + 1];
    const int i = blockIdx.x, c = blockIdx.y;
    const size_t base = (size_t)i * G.ny * G.nz;
    const R* src = in.c[c] + base;
    const uint8_t* ids = mid + base;
    conv_twiddles(tw, tw_g + G.ly.tw, G.ny + G.nz);
    if (mats) {
        for (int q = threadIdx.x; q <= nmat; q += blockDim.x) sMs[q] = (q > 0 && (mats[q - 1].flags & MF_FM)) ? mats[q - 1].Ms : R(0.);
        __syncthreads();
    }
    // row 2q as the real part, row 2q + 1 as the imaginary part
    const int ny = G.ny, nz = G.nz, nzc = G.nzc, pitch = G.pitch;
    struct In { R v0, v1; uint8_t i0, i1; };
    conv_items4<In>(G.pairs * nz,
                    [&](int it) {
                        const int q = G.dnz.div(it), e0 = 2 * q * nz + (it - q * nz);
                        const bool two = 2 * q + 1 < ny;
                        In r{src[e0], R(0.), 0, 0};
                        if (two) r.v1 = src[e0 + nz];
                        if (mats) { r.i0 = ids[e0]; if (two) r.i1 = ids[e0 + nz]; }
                        return r;
                    },
                    [&](int it, In r) {
                        const int q = G.dnz.div(it);
                        if (mats) {
                            const R m0 = sMs[r.i0], m1 = sMs[r.i1];
                            r.v0 = m0 != R(0.) ? m0 * r.v0 : R(0.);
                            r.v1 = m1 != R(0.) ? m1 * r.v1 : R(0.);
                        }
                        a[q * pitch + (it - q * nz)] = C{r.v0, r.v1};
                    });
    cp_async_wait_all();
    __syncthreads();
    C* z = conv_fft<false, R>(a, b, G.lz, G.pairs, G.dpairs, 1, pitch, tw + ny);
    C* y = z == a ? b : a;
    // the two rows' half spectra
    for (int it = threadIdx.x; it < G.pairs * nzc; it += blockDim.x) {
        const int q = G.dnzc.div(it), k = it - q * nzc;
        const C p = z[q * pitch + k], r = z[q * pitch + (k == 0 ? 0 : nz - k)];
        y[2 * q * nzc + k] = C{R(0.5) * (p.x + r.x), R(0.5) * (p.y - r.y)};
        if (2 * q + 1 < ny) y[(2 * q + 1) * nzc + k] = C{R(0.5) * (p.y + r.y), R(0.5) * (r.x - p.x)};
    }
    __syncthreads();
    y = conv_fft<false, R>(y, z, G.ly, nzc, G.dnzc, nzc, 1, tw);
    C* out = spec + (size_t)c * G.nk + (size_t)i * G.cols;
    for (int it = threadIdx.x; it < G.cols; it += blockDim.x) out[it] = y[it];
}

// tensor spectra of the form: FP64 nine complex (Axyz Ayzx Azxy Bxyz Byzx Bzxy
// Byxz Bzyx Bxzy), FP32 six real (N_xx N_yy N_zz N_xy N_yz N_zx)
template <class R> struct conv_tensor { using type = double2; };
template <> struct conv_tensor<float> { using type = float; };
template <class R> using ConvTensor = typename conv_tensor<R>::type;

// H_k = s N_k . M_k at point k; v holds the three components `g` words apart
__device__ __forceinline__ void conv_mul(const float* __restrict__ N, long nk, size_t k, float s, float2* v, int g) {
    const float2 mx = v[0], my = v[g], mz = v[2 * g];
    const float nxx = __ldg(N + k), nyy = __ldg(N + nk + k), nzz = __ldg(N + 2 * nk + k);
    const float nxy = __ldg(N + 3 * nk + k), nyz = __ldg(N + 4 * nk + k), nzx = __ldg(N + 5 * nk + k);
    v[0] = float2{s * (mx.x * nxx + my.x * nxy + mz.x * nzx), s * (mx.y * nxx + my.y * nxy + mz.y * nzx)};
    v[g] = float2{s * (my.x * nyy + mz.x * nyz + mx.x * nxy), s * (my.y * nyy + mz.y * nyz + mx.y * nxy)};
    v[2 * g] = float2{s * (mz.x * nzz + mx.x * nzx + my.x * nyz), s * (mz.y * nzz + mx.y * nzx + my.y * nyz)};
}
__device__ __forceinline__ void conv_mul(const double2* __restrict__ N, long nk, size_t k, double s, double2* v, int g) {
    const double2 mx = v[0], my = v[g], mz = v[2 * g];
    double2 n[9];
#pragma unroll
    for (int t = 0; t < 9; t++) n[t] = __ldg(N + t * nk + k);
    const double2 hx = cadd_(cadd_(cmul_(mx, n[0]), cmul_(my, n[3])), cmul_(mz, n[8]));
    const double2 hy = cadd_(cadd_(cmul_(my, n[1]), cmul_(mz, n[4])), cmul_(mx, n[6]));
    const double2 hz = cadd_(cadd_(cmul_(mz, n[2]), cmul_(mx, n[5])), cmul_(my, n[7]));
    v[0] = double2{s * hx.x, s * hx.y}; v[g] = double2{s * hy.x, s * hy.y}; v[2 * g] = double2{s * hz.x, s * hz.y};
}

// Block: columns g0 .. g0 + g - 1 of all three components, in place;
// s = -1 / (dx dy dz).
template <class R>
static __global__ void __launch_bounds__(kConvThreads, kConvXBlocks<R>) k_conv_x(const __grid_constant__ ConvGeom G, const Cx<R>* __restrict__ tw_g,
                                                        const ConvTensor<R>* __restrict__ N, R s, Cx<R>* __restrict__ spec) {
    using C = Cx<R>;
    GF_EXTERN_SMEM(unsigned char, smem_raw);
    const int g = G.g, lines = 3 * g, words = lines * G.nx;
    C* a = reinterpret_cast<C*>(smem_raw);
    C* b = a + words;
    C* tw = b + words;
    const int g0 = blockIdx.x * g, cols = G.cols;
    conv_twiddles(tw, tw_g + G.lx.tw, G.nx);
    // line q: component q / g, column g0 + q % g (past the last column it
    // repeats that column, and is not stored)
    for (int it = threadIdx.x; it < words; it += blockDim.x) {
        const int x = G.dlines.div(it), q = it - x * lines, c = G.dg.div(q);
        conv_copy(a + it, spec + (size_t)c * G.nk + (size_t)x * cols + min(g0 + q - c * g, cols - 1));
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    C* f = conv_fft<false, R>(a, b, G.lx, lines, G.dlines, lines, 1, tw);
    for (int it = threadIdx.x; it < g * G.nx; it += blockDim.x) {
        const int x = G.dg.div(it), q = it - x * g;
        conv_mul(N, G.nk, (size_t)x * cols + min(g0 + q, cols - 1), s, f + x * lines + q, g);
    }
    __syncthreads();
    f = conv_fft<true, R>(f, f == a ? b : a, G.lx, lines, G.dlines, lines, 1, tw);
    for (int it = threadIdx.x; it < words; it += blockDim.x) {
        const int x = G.dlines.div(it), q = it - x * lines;
        const int c = G.dg.div(q), col = g0 + q - c * g;
        if (col < cols) spec[(size_t)c * G.nk + (size_t)x * cols + col] = f[it];
    }
}

// Block (plane i, component c): the half spectrum back to H.
template <class R>
static __global__ void __launch_bounds__(kConvThreads, kConvPlaneBlocks<R>) k_conv_inv(const __grid_constant__ ConvGeom G, const Cx<R>* __restrict__ tw_g,
                                                          const Cx<R>* __restrict__ spec, F3T<R> out) {
    using C = Cx<R>;
    GF_EXTERN_SMEM(unsigned char, smem_raw);
    C* a = reinterpret_cast<C*>(smem_raw);
    C* b = a + G.plane;
    C* tw = b + G.plane;
    const int i = blockIdx.x, c = blockIdx.y;
    const int pitch = G.pitch, nz = G.nz, nzc = G.nzc, ny = G.ny;
    conv_twiddles(tw, tw_g + G.ly.tw, G.ny + G.nz);
    const C* in = spec + (size_t)c * G.nk + (size_t)i * G.cols;
    for (int it = threadIdx.x; it < G.cols; it += blockDim.x) conv_copy(a + it, in + it);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    C* y = conv_fft<true, R>(a, b, G.ly, nzc, G.dnzc, nzc, 1, tw);
    C* z = y == a ? b : a;
    // rows 2q and 2q + 1 as one complex row: A + i B with both extended by
    // their conjugates; k = 0 and the Nyquist point of a real row are real
    for (int it = threadIdx.x; it < G.pairs * nzc; it += blockDim.x) {
        const int q = G.dnzc.div(it), k = it - q * nzc;
        const C A = y[2 * q * nzc + k], B = 2 * q + 1 < ny ? y[(2 * q + 1) * nzc + k] : C{R(0.), R(0.)};
        if (k == 0 || 2 * k == nz) z[q * pitch + k] = C{A.x, B.x};
        else {
            z[q * pitch + k] = C{A.x - B.y, A.y + B.x};
            z[q * pitch + nz - k] = C{A.x + B.y, B.x - A.y};
        }
    }
    __syncthreads();
    z = conv_fft<true, R>(z, y, G.lz, G.pairs, G.dpairs, 1, pitch, tw + ny);
    R* dst = out.c[c] + (size_t)i * ny * nz;
    for (int it = threadIdx.x; it < ny * nz; it += blockDim.x) {
        const int row = G.dnz.div(it), k = it - row * nz;
        const C v = z[(row >> 1) * pitch + k];
        dst[it] = (row & 1) ? v.y : v.x;
    }
}

// ---- host side ----

// radices of length n: the fewest passes, then the smallest largest radix;
// false when n has another prime factor than 2, 3, 5
inline void conv_split(int n, int from, int depth, int* cur, int& best, int& top, int* out) {
    static const int rads[6] = {8, 6, 5, 4, 3, 2};
    if (n == 1) {
        int mx = 1;
        for (int q = 0; q < depth; q++) mx = std::max(mx, cur[q]);
        if (depth < best || (depth == best && mx < top)) {
            best = depth; top = mx;
            for (int q = 0; q < depth; q++) out[q] = cur[q];
        }
        return;
    }
    if (depth >= best || depth >= kConvMaxPass) return;
    for (int q = from; q < 6; q++)
        if (n % rads[q] == 0) {
            cur[depth] = rads[q];
            conv_split(n / rads[q], q, depth + 1, cur, best, top, out);
        }
}
inline bool conv_len(int n, ConvLen& L) {
    L.n = n; L.np = 0;
    if (n < 1 || n > kConvMaxSide) return false;
    if (n > 1) {
        int cur[kConvMaxPass] = {}, best = kConvMaxPass + 1, top = 0;
        conv_split(n, 0, 0, cur, best, top, L.rad);
        if (best > kConvMaxPass) return false;
        L.np = best;
    }
    int l = 1;
    for (int p = 0; p < L.np; p++) { L.l[p] = l; L.dl[p] = conv_div(l); l *= L.rad[p]; }
    return true;
}
template <class R>
inline size_t conv_plane_smem(const ConvGeom& g) { return ((size_t)2 * g.plane + g.ny + g.nz) * sizeof(Cx<R>); }
template <class R>
inline size_t conv_x_smem(const ConvGeom& g) { return ((size_t)6 * g.g * g.nx + g.nx) * sizeof(Cx<R>); }

// Geometry for a grid on a device of `sms` SMs, or false when the transforms
// do not cover it (another prime factor, or buffers beyond the shared memory
// of a block).
template <class R>
inline bool conv_geom(int nx, int ny, int nz, int sms, ConvGeom& g) {
    g = ConvGeom{};
    g.nx = nx; g.ny = ny; g.nz = nz; g.nzc = nz / 2 + 1;
    g.n = (long)nx * ny * nz;
    g.cols = ny * g.nzc;
    g.nk = (long)nx * g.cols;
    if (!conv_len(nx, g.lx) || !conv_len(ny, g.ly) || !conv_len(nz, g.lz)) return false;
    g.lx.tw = 0; g.ly.tw = nx; g.lz.tw = nx + ny;
    g.pairs = (ny + 1) / 2;
    g.pitch = nz | 1;
    g.plane = std::max(g.pairs * g.pitch, g.cols);
    if (conv_plane_smem<R>(g) > kConvMaxSmem) return false;
    g.dpairs = conv_div(g.pairs); g.dnz = conv_div(nz); g.dnzc = conv_div(g.nzc);
    // columns per block: 128-byte rows where two such blocks fit on an SM,
    // fewer (never below 32 bytes) for long x, and fewer on films whose blocks
    // would be less than three for two SMs: between one and 1.5 per SM some
    // SMs run two of the long blocks while the others wait (FP32 ms per step,
    // at least 1 / 1.5 / 2 per SM: 108x120x24 0.154 / 0.148 / 0.149, 72x100x48
    // 0.171 / 0.162 / 0.162; FP64 120x90x20 0.149 / 0.146 / 0.161, whose
    // 32-byte rows cost more than they spread)
    int c = 128 / (int)sizeof(Cx<R>);
    const int least = 32 / (int)sizeof(Cx<R>);
    auto bytes = [&](int v) { return ((size_t)6 * v + 1) * nx * sizeof(Cx<R>); };
    while (c > least && (bytes(c) > 100 * 1024 || 2l * ((g.cols + c - 1) / c) < 3l * sms)) c /= 2;
    if (bytes(c) > kConvMaxSmem) return false;
    g.g = c;
    g.groups = (g.cols + c - 1) / c;
    g.dlines = conv_div(3 * c); g.dg = conv_div(c);
    // the divisions by reciprocal cover indices below 2^20
    return (long)g.plane < (1l << 20) && (long)3 * c * nx < (1l << 20) && (long)ny * nz < (1l << 20);
}

// plane blocks that fit on an SM by their shared memory
template <class R>
inline int conv_plane_fit(const ConvGeom& g) { return (int)((size_t)227 * 1024 / (conv_plane_smem<R>(g) + 1024)); }

// Where the engine's transforms beat cuFFT's in a stage, with or without
// elastodynamics (the convolution follows the join of a stage's branches, so
// it runs alone in both).  ms per step, own / cuFFT, FP32 and FP64, of films
// of ferromagnets alone:
//  * films up to 2^19 cells: 32x32x8 0.063 / 0.078 and 0.065 / 0.088, 64x64x16
//    0.075 / 0.088 and 0.082 / 0.109, 120x90x20 0.120 / 0.126 and 0.150 /
//    0.164, 128x128x32 0.189 / 0.204 and 0.284 / 0.313; beyond, 192x192x24
//    0.320 / 0.299 and 0.530 / 0.537;
//  * x in three passes of at most 256 points (an x block of four passes or of
//    two per SM is long): 250x150x8 0.173 / 0.165 and 0.276 / 0.264, 512x64x8
//    0.168 / 0.137 and 0.259 / 0.205;
//  * planes that leave an SM three blocks in FP32, two in FP64, or that are all
//    resident at once: 48x320x32 0.196 / 0.223 and 0.277 / 0.328, but 64x256x32
//    (FP64, 192 blocks at one per SM) 0.358 / 0.307;
//  * planes of more than 2048 points only where there is about one per SM:
//    18x256x18 0.106 / 0.099 and 0.124 / 0.117, 24x384x32 0.182 / 0.170 and
//    0.232 / 0.220, 24x200x50 0.170 / 0.147 and 0.216 / 0.199;
//  * FP32: y of four passes only up to 2^17 cells: 90x135x8 0.095 / 0.109, but
//    100x300x15 0.200 / 0.176 (FP64 0.331 / 0.352).
// With elastodynamics the same lines hold: 90x120x40 0.284 / 0.294 and 0.423 /
// 0.443, but 192x192x24 0.500 / 0.483 and 0.824 / 0.812.  Slower inside the
// lines: FP32 108x120x24 0.148 / 0.145, FP64 240x90x24 0.307 / 0.302.
template <class R>
inline bool conv_pays(const ConvGeom& g, int sms) {
    constexpr bool f32 = sizeof(R) == 4;
    const int fit = conv_plane_fit<R>(g);
    const long blocks = 3l * g.nx;
    return g.n <= (1l << 19) && g.nx <= 256 && g.lx.np <= 3 && (fit >= (f32 ? 3 : 2) || blocks <= (long)fit * sms) &&
           (g.plane <= 2048 || 10 * blocks >= 9l * sms) && (!f32 || g.ly.np <= 3 || g.n <= (1l << 17));
}

// The same for the discrete adjoint, which launches its stages one by one:
// three launches in place of cuFFT's eight to twelve gain more there.  ms per
// step of a forward and backward run of magnetoelastic films, own / cuFFT,
// FP32 and FP64: 32x32x8 0.62 / 0.79 and 0.60 / 0.80, 108x120x24 1.30 / 1.39
// and 1.52 / 1.72, 192x192x24 2.18 / 2.32 and 3.31 / 3.47, FP32 256x256x32 4.35
// / 4.50; beyond the lines 512x512x8 4.90 / 4.78 and 8.3 / 7.7, FP64 256x256x32
// 7.70 / 6.85, one plane block per SM (27x384x45 FP32) 1.86 / 1.82.
template <class R>
inline bool adj_conv_pays(const ConvGeom& g) {
    return g.n <= (sizeof(R) == 4 ? (1l << 21) : (1l << 20)) && g.nx <= 256 && conv_plane_fit<R>(g) >= (sizeof(R) == 4 ? 2 : 1);
}

}  // namespace gf
