// Register-tiled fp32 products for what the tensor-core kernels do not take at fp32 precision: deltaX of channel counts that
// are no multiple of 8 (stride 1) or 32 (strides), and batched matrix products of ragged sizes.
//
// Bound: FMA issue with the operand reads from shared memory close behind (a step of a 128 x 64 tile is 64 clocks of FMAs and some
// 40 of reads).  Of 74 TFLOP/s it reaches 42 with 128 x 128 tiles (64 x 56 x 56, 100 -> 128 channels 3x3) and, with 128 x 64 tiles,
// 32 counting idle columns: 18 of use at 36 of 64 columns (50 x 35 x 29, 100 -> 36).
//
// A CTA of 256 threads computes BM x BN outputs, TM x TN per thread, from 16 reduction steps staged in shared memory at a time.
// Both operands lie k-major there ([16][BM], [16][BN]), so a thread reads its TM + TN operands of a step as 16-byte words (the A
// words are broadcast within a warp, the B words consecutive) and issues TM * TN FMAs on them,
// two columns per instruction (fma.rn.f32x2: each half is an ordinary fp32 FMA, so the sum of an element is the same chain of
// FMAs in ascending k as one thread per element would form).  The next tile is loaded into registers while the current one is
// multiplied, and the shared tiles are double-buffered: one barrier per 16 steps.  An operand whose memory runs along k is
// transposed on its way into shared memory; its columns are exchanged in blocks of 8 by the 4-step group of k
// (column ^ 8 * (k / 4)), which spreads the 4 x 8 words a warp stores over all 32 banks.
//
// What is multiplied is described by a policy P (by value, in the kernel's parameters):
//   P::kAk, P::kBk     operand runs along k in memory (else along its rows / columns)
//   cta()              block-level state of this CTA: k-tiles [it0, it1) and whatever the loads need; false: nothing to do
//   load_a / load_b    one 16-byte word of a tile, zero outside the problem
//   store              four consecutive outputs of a row
//   P::kSkip           a row may have no operand in a whole tile (a filter tap outside the output): its A words are zeros, and
//                      meets() says so.  Zeros add nothing unless B holds an Inf or NaN there, which leaves a NaN: a CTA that
//                      finds one among its sums forms them once more, row by row without the tiles a row does not meet.
#pragma once
#include "dependent_launch.cuh"
#include "fast_div.cuh"
#include <type_traits>

namespace alpha {

constexpr int kGemmThreads = 256, kGemmBK = 16;

__device__ __forceinline__ void ffma2(unsigned long long& d, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float x, float y)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& x, float& y)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}

// Word w of a tile of 16 steps x COLS columns.  Along k: column w / 4, steps 4 * (w % 4) ...; else step w / (COLS / 4), four columns.
template <int COLS, bool KC> __device__ __forceinline__ int word_col(int w) { return KC ? w >> 2 : (w % (COLS / 4)) * 4; }
template <int COLS, bool KC> __device__ __forceinline__ int word_k(int w) { return KC ? (w & 3) * 4 : w / (COLS / 4); }

template <int COLS, bool KC>
__device__ __forceinline__ void put_word(float* tile, int w, const float4& v)
{
    const int c = word_col<COLS, KC>(w), k = word_k<COLS, KC>(w);
    float* p = tile + k * COLS + (c ^ ((k >> 2) * 8));
    if (KC) {
        p[0] = v.x; p[COLS] = v.y; p[2 * COLS] = v.z; p[3 * COLS] = v.w;
    } else {
        *reinterpret_cast<float4*>(p) = v;
    }
}

template <int BM, int BN, int TM, int TN, class P>
__global__ void __launch_bounds__(kGemmThreads, 2) gemm_f32_kernel(const P p)
{
    static_assert((BM / TM) * (BN / TN) == kGemmThreads && TN % 4 == 0 && TM % 4 == 0 && BM >= 32 && BN >= 32, "tile shape");
    constexpr int WA = BM * 4, WB = BN * 4;                       // 16-byte words of a tile
    constexpr int NA = WA / kGemmThreads, NB = (WB + kGemmThreads - 1) / kGemmThreads;
    static_assert(WA % kGemmThreads == 0, "A words");
    __shared__ __align__(16) float As[2][kGemmBK * BM];
    __shared__ __align__(16) float Bs[2][kGemmBK * BN];
    __shared__ bool met[2][P::kSkip ? BM : 1];
    const int tid = threadIdx.x, tx = tid % (BN / TN), ty = tid / (BN / TN);

    grid_dependency_wait();
    grid_dependency_trigger();
    typename P::Cta c;
    if (!p.cta(c, BM, BN)) return;                                // uniform for the CTA
    typename P::RowA ra[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) ra[i] = p.row_a(c, word_col<BM, P::kAk>(tid + i * kGemmThreads));

    unsigned long long acc[TM][TN / 2];
    auto form_sums = [&](auto by_row_) {
        constexpr bool by_row = decltype(by_row_)::value;
#pragma unroll
        for (int y = 0; y < TM; ++y)
#pragma unroll
            for (int x = 0; x < TN / 2; ++x) acc[y][x] = 0ull;
        float4 va[NA], vb[NB];
        bool vm[by_row ? NA : 1];
        auto fetch = [&](int it) {
            const typename P::Step st = p.step(c, it);
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                va[i] = p.load_a(c, st, ra[i], word_col<BM, P::kAk>(tid + i * kGemmThreads), word_k<BM, P::kAk>(tid + i * kGemmThreads));
                if constexpr (by_row) vm[i] = p.meets(c, st, ra[i]);
            }
#pragma unroll
            for (int i = 0; i < NB; ++i)
                if (WB % kGemmThreads == 0 || tid + i * kGemmThreads < WB)
                    vb[i] = p.load_b(c, st, word_col<BN, P::kBk>(tid + i * kGemmThreads), word_k<BN, P::kBk>(tid + i * kGemmThreads));
        };
        auto stage = [&](int buf) {
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                put_word<BM, P::kAk>(As[buf], tid + i * kGemmThreads, va[i]);
                if constexpr (by_row) met[buf][word_col<BM, P::kAk>(tid + i * kGemmThreads)] = vm[i];   // (words of a row agree)
            }
#pragma unroll
            for (int i = 0; i < NB; ++i)
                if (WB % kGemmThreads == 0 || tid + i * kGemmThreads < WB) put_word<BN, P::kBk>(Bs[buf], tid + i * kGemmThreads, vb[i]);
        };
        if (c.it0 < c.it1) {
            fetch(c.it0);
            stage(0);
        }
        __syncthreads();
        int buf = 0;
        for (int it = c.it0; it < c.it1; ++it) {
            if (it + 1 < c.it1) fetch(it + 1);
#pragma unroll(by_row ? 1 : kGemmBK)
            for (int k = 0; k < kGemmBK; ++k) {
                const int x8 = (k >> 2) * 8;
                float a[TM];
                unsigned long long b[TN / 2];
#pragma unroll
                for (int y = 0; y < TM; y += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(&As[buf][k * BM + ((ty * TM + y) ^ x8)]);
                    a[y] = t.x; a[y + 1] = t.y; a[y + 2] = t.z; a[y + 3] = t.w;
                }
                // columns tx * 4 ... of each group of BN / (TN / 4) columns
#pragma unroll
                for (int x = 0; x < TN; x += 4) {
                    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&Bs[buf][k * BN + (((x / 4) * (BN * 4 / TN) + tx * 4) ^ x8)]);
                    b[x / 2] = t.x; b[x / 2 + 1] = t.y;
                }
#pragma unroll
                for (int y = 0; y < TM; ++y) {
                    if constexpr (by_row)
                        if (!met[buf][ty * TM + y]) continue;
                    const unsigned long long aa = pack2(a[y], a[y]);
#pragma unroll
                    for (int x = 0; x < TN / 2; ++x) ffma2(acc[y][x], aa, b[x]);
                }
            }
            if (it + 1 < c.it1) stage(buf ^ 1);   // the other buffer was last read before the previous barrier
            __syncthreads();
            buf ^= 1;
        }
    };
    form_sums(std::false_type{});
    if constexpr (P::kSkip) {
        bool nan = false;
#pragma unroll
        for (int y = 0; y < TM; ++y)
#pragma unroll
            for (int x = 0; x < TN / 2; ++x) {
                float u, v;
                unpack2(acc[y][x], u, v);
                nan = nan || u != u || v != v;
            }
        if (__syncthreads_or(nan)) form_sums(std::true_type{});
    }
#pragma unroll
    for (int y = 0; y < TM; ++y) {
        const typename P::RowC rc = p.row_c(c, ty * TM + y);
#pragma unroll
        for (int x = 0; x < TN; x += 4) {
            float4 o;
            unpack2(acc[y][x / 2], o.x, o.y);
            unpack2(acc[y][x / 2 + 1], o.z, o.w);
            p.store(c, rc, (x / 4) * (BN * 4 / TN) + tx * 4, o);
        }
    }
}

// deltaX of any stride as an implicit GEMM: rows = the pixels of one stride phase (py, px), which all receive the same filter
// taps, columns = input channels, reduction = those taps x output channels (tap-major), in ksplit parts.  A launch computes `parts` of
// them from part0 on, blockIdx.z = phase * parts + part, each into its own copy of deltaX (out + part * size), every element of which
// some phase writes; or, without memory for copies, one part that is added to what `out` holds (DxGemm<true>, a kernel of its own: the
// test and the load in the epilogue of every launch cost 7 % of a small layer): the same sums in the same order.
struct DxProblem {
    static constexpr bool kAk = true, kBk = false, kSkip = true;
    const float* dY; const float* W; float* out;
    int N, IH, IW, IC, FH, FW, OH, OW, OC, sh, sw, ph, pw;
    int nsw;                       // phases along a row: min(sw, IW)
    int ksplit, parts, part0;
    int kt, y0, z0;                // kt = 16-step tiles per tap; y0 = column tile of blockIdx.y == 0, z0 = phase * parts + part of blockIdx.z == 0
    size_t size;                   // elements of deltaX
    FastDiv by_kt;
    struct Cta { int m0, n0, rows, it0, it1, A, B, py, px, ry, rx, qy, qx, Ux; float* out; };
    struct RowA { int n, a, b; };  // n < 0: past the last row
    struct Step { int fh, fw, u, v, k0; };
    struct RowC { float* p; };

    __device__ bool cta(Cta& c, int BM, int BN) const
    {
        const int z = z0 + static_cast<int>(blockIdx.z), phase = z / parts, copy = z - phase * parts, sp = part0 + copy;
        c.py = phase / nsw; c.px = phase - c.py * nsw;
        c.A = (IH - c.py + sh - 1) / sh; c.B = (IW - c.px + sw - 1) / sw;
        c.rows = N * c.A * c.B;
        c.m0 = static_cast<int>(blockIdx.x) * BM; c.n0 = (y0 + static_cast<int>(blockIdx.y)) * BN;
        if (c.m0 >= c.rows) return false;
        c.ry = (c.py + ph) % sh; c.rx = (c.px + pw) % sw;
        c.qy = (c.py + ph - c.ry) / sh; c.qx = (c.px + pw - c.rx) / sw;
        const int Uy = c.ry < FH ? (FH - c.ry + sh - 1) / sh : 0;
        c.Ux = c.rx < FW ? (FW - c.rx + sw - 1) / sw : 0;
        const int its = Uy * c.Ux * kt, per = (its + ksplit - 1) / ksplit;
        c.it0 = sp * per < its ? sp * per : its;
        c.it1 = c.it0 + per < its ? c.it0 + per : its;
        c.out = out + static_cast<size_t>(copy) * size;
        return true;
    }
    __device__ RowA row_a(const Cta& c, int m) const
    {
        const int r = c.m0 + m;
        if (r >= c.rows) return RowA{-1, 0, 0};
        const int n = r / (c.A * c.B), q = r - n * (c.A * c.B), a = q / c.B;
        return RowA{n, a, q - a * c.B};
    }
    __device__ Step step(const Cta& c, int it) const
    {
        const int t = static_cast<int>(by_kt.div(static_cast<unsigned>(it)));
        Step s;
        s.k0 = (it - t * kt) * kGemmBK;
        s.u = t / c.Ux; s.v = t - s.u * c.Ux;
        s.fh = c.ry + sh * s.u; s.fw = c.rx + sw * s.v;
        return s;
    }
    __device__ bool meets(const Cta& c, const Step& s, const RowA& r) const
    {
        return r.n >= 0 && static_cast<unsigned>(r.a + c.qy - s.u) < static_cast<unsigned>(OH) && static_cast<unsigned>(r.b + c.qx - s.v) < static_cast<unsigned>(OW);
    }
    __device__ float4 load_a(const Cta& c, const Step& s, const RowA& r, int, int k) const
    {
        const int oh = r.a + c.qy - s.u, ow = r.b + c.qx - s.v, oc = s.k0 + k;
        if (r.n < 0 || oc >= OC || static_cast<unsigned>(oh) >= static_cast<unsigned>(OH) || static_cast<unsigned>(ow) >= static_cast<unsigned>(OW))
            return make_float4(0.f, 0.f, 0.f, 0.f);
        return __ldg(reinterpret_cast<const float4*>(dY + ((static_cast<size_t>(r.n) * OH + oh) * OW + ow) * OC + oc));
    }
    __device__ float4 load_b(const Cta& c, const Step& s, int col, int k) const
    {
        const int oc = s.k0 + k, ic = c.n0 + col;
        if (oc >= OC || ic >= IC) return make_float4(0.f, 0.f, 0.f, 0.f);
        return __ldg(reinterpret_cast<const float4*>(W + ((static_cast<size_t>(oc) * FH + s.fh) * FW + s.fw) * IC + ic));
    }
    __device__ RowC row_c(const Cta& c, int m) const
    {
        const RowA r = row_a(c, m);
        if (r.n < 0) return RowC{nullptr};
        return RowC{c.out + ((static_cast<size_t>(r.n) * IH + (r.a * sh + c.py)) * IW + (r.b * sw + c.px)) * IC};
    }
};
template <bool ADD>
struct DxGemm : DxProblem {
    __device__ void store(const Cta& c, const RowC& r, int col, const float4& o) const
    {
        if (!r.p || c.n0 + col >= IC) return;
        float4* p = reinterpret_cast<float4*>(r.p + c.n0 + col);
        if (ADD) {
            const float4 a = *p;
            *p = make_float4(a.x + o.x, a.y + o.y, a.z + o.z, a.w + o.w);
        } else {
            *p = o;
        }
    }
};

// The tiles of a deltaW that hold an Inf or NaN, once more and in fp32: rows = output channels, columns = deltaW's taps x input
// channels, reduction = pixels in ascending order; a CTA whose tile is finite returns at once.  The tensor kernel's pixel tiles may
// reach past the output, where deltaY is zero but X can be a pixel of the image: finite pixels add nothing there, an Inf or NaN would
// make deltaW NaN at taps that never meet it.  Looking at a finite deltaW costs about 2 us (100 x 3 x 3 x 36).
struct DwRepair {
    static constexpr bool kAk = false, kBk = false, kSkip = false;
    const float *dY, *X; float* dW;
    int IH, IW, IC, OC, FW, sh, sw, ph, pw, L, P;   // L = floats of a row of deltaW, P = output pixels
    FastDiv by_IC, by_FW, by_OW, by_OH;
    struct Cta { int m0, n0, it0, it1; };
    struct RowA {};
    struct Step { int k0; };
    struct RowC { float* p; };

    __device__ bool cta(Cta& c, int BM, int BN) const
    {
        c.m0 = static_cast<int>(blockIdx.x) * BM; c.n0 = static_cast<int>(blockIdx.y) * BN;
        c.it0 = 0; c.it1 = (P + kGemmBK - 1) / kGemmBK;
        float z = 0.f;
        for (int i = threadIdx.x; i < BM * BN / 4; i += kGemmThreads) {
            const int oc = c.m0 + i / (BN / 4), col = c.n0 + i % (BN / 4) * 4;
            if (oc >= OC || col >= L) continue;
            const float4 v = *reinterpret_cast<const float4*>(dW + static_cast<size_t>(oc) * L + col);
            z += v.x * 0.f + v.y * 0.f + v.z * 0.f + v.w * 0.f;
        }
        return __syncthreads_or(z != 0.f) != 0;
    }
    __device__ RowA row_a(const Cta&, int) const { return RowA{}; }
    __device__ bool meets(const Cta&, const Step&, const RowA&) const { return true; }
    __device__ Step step(const Cta&, int it) const { return Step{it * kGemmBK}; }
    __device__ float4 load_a(const Cta& c, const Step& s, const RowA&, int m, int k) const
    {
        const int px = s.k0 + k, oc = c.m0 + m;
        if (px >= P || oc >= OC) return make_float4(0.f, 0.f, 0.f, 0.f);
        return __ldg(reinterpret_cast<const float4*>(dY + static_cast<size_t>(px) * OC + oc));
    }
    __device__ float4 load_b(const Cta& c, const Step& s, int col, int k) const
    {
        const int px = s.k0 + k, q = c.n0 + col;
        if (px >= P || q >= L) return make_float4(0.f, 0.f, 0.f, 0.f);
        unsigned t, ic, fh, fw, n, oh, ow;
        by_IC.divmod(static_cast<unsigned>(q), t, ic);
        by_FW.divmod(t, fh, fw);
        by_OW.divmod(static_cast<unsigned>(px), t, ow);
        by_OH.divmod(t, n, oh);
        const int ih = static_cast<int>(oh) * sh + static_cast<int>(fh) - ph, iw = static_cast<int>(ow) * sw + static_cast<int>(fw) - pw;
        if (static_cast<unsigned>(ih) >= static_cast<unsigned>(IH) || static_cast<unsigned>(iw) >= static_cast<unsigned>(IW)) return make_float4(0.f, 0.f, 0.f, 0.f);
        return __ldg(reinterpret_cast<const float4*>(X + ((static_cast<size_t>(n) * IH + ih) * IW + iw) * IC + ic));
    }
    __device__ RowC row_c(const Cta& c, int m) const { return RowC{c.m0 + m < OC ? dW + static_cast<size_t>(c.m0 + m) * L : nullptr}; }
    __device__ void store(const Cta& c, const RowC& r, int col, const float4& o) const
    {
        if (r.p && c.n0 + col < L) *reinterpret_cast<float4*>(r.p + c.n0 + col) = o;
    }
};

// C[b] = A[b] * B[b] over N x M outputs and K steps, with row pitches.  A_KC: A[b] is [N][lda] (else [K][lda], the transposed
// form); B_KC: B[b] is [M][ldb] (else [K][ldb]).  Pitches are multiples of 4 and every matrix starts on a 16-byte boundary;
// words are loaded whole where they start inside the matrix, and what they hold past N, M or K is replaced by zeros.
template <bool A_KC, bool B_KC>
struct BatchGemm {
    static constexpr bool kAk = A_KC, kBk = B_KC, kSkip = false;
    const float *A, *B; float* C;
    int N, M, K, lda, ldb, ldc;
    size_t strA, strB, strC;
    struct Cta { int m0, n0, it0, it1; const float *A, *B; float* C; };
    struct RowA {};
    struct Step { int k0; };
    struct RowC { float* p; };

    __device__ bool cta(Cta& c, int BM, int BN) const
    {
        c.m0 = static_cast<int>(blockIdx.y) * BM; c.n0 = static_cast<int>(blockIdx.x) * BN;
        c.it0 = 0; c.it1 = (K + kGemmBK - 1) / kGemmBK;
        c.A = A + blockIdx.z * strA; c.B = B + blockIdx.z * strB; c.C = C + blockIdx.z * strC;
        return true;
    }
    __device__ RowA row_a(const Cta&, int) const { return RowA{}; }
    __device__ bool meets(const Cta&, const Step&, const RowA&) const { return true; }
    __device__ Step step(const Cta&, int it) const { return Step{it * kGemmBK}; }
    // the word of four consecutive elements that starts at (row, col): elements at col + i >= cols are zero
    __device__ static float4 word(const float* base, int ld, int row, int rows, int col, int cols)
    {
        if (row >= rows || col >= cols) return make_float4(0.f, 0.f, 0.f, 0.f);
        float4 v = __ldg(reinterpret_cast<const float4*>(base + static_cast<size_t>(row) * ld + col));
        if (col + 3 >= cols) {
            if (col + 1 >= cols) v.y = 0.f;
            if (col + 2 >= cols) v.z = 0.f;
            v.w = 0.f;
        }
        return v;
    }
    __device__ float4 load_a(const Cta& c, const Step& s, const RowA&, int m, int k) const
    {
        return A_KC ? word(c.A, lda, c.m0 + m, N, s.k0 + k, K) : word(c.A, lda, s.k0 + k, K, c.m0 + m, N);
    }
    __device__ float4 load_b(const Cta& c, const Step& s, int n, int k) const
    {
        return B_KC ? word(c.B, ldb, c.n0 + n, M, s.k0 + k, K) : word(c.B, ldb, s.k0 + k, K, c.n0 + n, M);
    }
    __device__ RowC row_c(const Cta& c, int m) const { return RowC{c.m0 + m < N ? c.C + static_cast<size_t>(c.m0 + m) * ldc : nullptr}; }
    __device__ void store(const Cta& c, const RowC& r, int col, const float4& o) const
    {
        const int j = c.n0 + col;
        if (!r.p || j >= M) return;
        if (j + 3 < M) { *reinterpret_cast<float4*>(r.p + j) = o; return; }
        r.p[j] = o.x;
        if (j + 1 < M) r.p[j + 1] = o.y;
        if (j + 2 < M) r.p[j + 2] = o.z;
    }
};

// Tile for a product of `rows` x `cols` outputs, `copies` times: the shape whose launch is shortest, in FMAs of the busiest SM
// over the share of the FMA rate it reaches (a smaller tile reads more shared memory per FMA).
struct GemmTile { int bm, bn; bool planes = false; };
inline GemmTile pick_gemm_tile(long long rows, int cols, long long copies, int sms)
{
    static const struct { int bm, bn; double eff; } cand[] = {{128, 128, 1.0}, {128, 64, 0.9}, {64, 64, 0.8}, {128, 32, 0.7}};
    GemmTile best{0, 0};
    double best_t = 0;
    for (const auto& c : cand) {
        const double ctas = (double)((rows + c.bm - 1) / c.bm) * ((cols + c.bn - 1) / c.bn) * copies;
        const double t = (ctas > sms ? ctas / sms : 1.0) * c.bm * c.bn / c.eff;
        if (!best.bm || t < best_t) { best = GemmTile{c.bm, c.bn}; best_t = t; }
    }
    return best;
}

template <class P>
inline void launch_gemm_f32(const P& p, const GemmTile& t, dim3 grid, cudaStream_t stream)
{
    if (t.bn == 128) launch_after(gemm_f32_kernel<128, 128, 8, 8, P>, grid, kGemmThreads, 0, stream, p);
    else if (t.bn == 32) launch_after(gemm_f32_kernel<128, 32, 4, 4, P>, grid, kGemmThreads, 0, stream, p);
    else if (t.bm == 128) launch_after(gemm_f32_kernel<128, 64, 8, 4, P>, grid, kGemmThreads, 0, stream, p);
    else launch_after(gemm_f32_kernel<64, 64, 4, 4, P>, grid, kGemmThreads, 0, stream, p);
}

}  // namespace alpha
