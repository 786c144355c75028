// Products on the tensor cores at fp32 accuracy, gathering both operands from the tensors as they lie.
//
// An fp32 word is the exact sum of three bf16 words, x = h + m + l (8 bits of significand each: x rounded to nearest, what is left
// of it rounded, the rest, so that |m| <= 2^-8 |x| and |l| <= 2^-17 |x|), and of the nine products of two such sums the six that matter are
// formed by tcgen05.mma kind::f16: hh in one accumulator; hm, mh, mm, hl, lh, all below 2^-7 of it, in another.  What is dropped (ml, lm,
// ll) is below 2^-24 (1 + 2^-10) of a product, as much as an fp32 rounding, and of either sign (truncated words would leave 2^-21, always
// towards zero: 1.0078124 squared 4.7e-7 too small).
// The tensor core truncates as it adds to an accumulator, about 2^-24 of it an instruction, which over a long sum would cost more
// than fp32 FMAs do: after every 64 reduction steps (four instructions into the hh accumulator) the partial sum is added to running
// sums in registers, rounded to nearest, and the accumulator starts anew.  2-norm errors against 64 bits (operands in [0, 1) / N(0, 1); in
// brackets the FMA kernel, which keeps products of under 64 terms): 1 term 3.6e-8 / 3.5e-8 (2.5e-8), 16 4.5e-8 / 4.4e-8 (6.3e-8 / 7.3e-8), 64
// 8.7e-8 / 7.6e-8 (1.2e-7 / 1.5e-7), 513 9.1e-8 / 9.4e-8 (3.1e-7 / 4.1e-7), 20001 2.8e-7 / 3.4e-7 (2.2e-6 / 2.5e-6).
//
// Bound: 388 clocks of MMAs per 16 steps of a 128 x 128 tile, as much as the 3xTF32 kernels issue per step.  A stage of 32 steps takes
// 0.80 us (some 1450 clocks for the 776 of MMAs): the issue slots and shared memory accesses of the loads and splits, and the wait of
// fence.proxy.async for loads in flight.  With B split beforehand and copied by TMA 0.57 us.  2368 x 2048 x 2304: 195 -> 140 us, and the
// FMA kernel 640.
//
// A CTA of 576 threads forms 128 x BN outputs of a policy P, in stages of 32 steps:
//   warps 0-15  in two groups that take alternate stages, so that the loads of one are in flight while the other splits: load the words of
//               a stage, split them and store the planes of both operands in shared memory as the MMA reads them - rows of 32 steps where
//               the operand's memory runs along k (K-major), rows of 32 columns where it does not (MN-major; no transposition) - with the
//               64-byte swizzle; a warp's four rows of eight words are 256 consecutive bytes of a plane, half a warp's 128 all banks once.  They also add
//               up the flushed sums, a quarter of the columns each, and store the result.  96 registers a thread allow no more: with more
//               live words or sums they spill, and what spills goes to L2 (shared memory leaves no L1; 44 TFLOP/s).
//   warp 16     issues the MMAs.  The three planes of B are neighbouring rows (or column blocks) of one operand, so that h x [m l], m x [h m]
//               are one MMA each, and with BN = 64 also h x [h m l].
//   warp 17     where W is split beforehand (TMA_B), copies the three planes of a stage of B; half of the split work goes.
// hh accumulates in two column blocks in turn, so that one is read while the other fills.
// Where an operand is not the sum of its planes (below 2^-110 its last bits underflow them), or a sum comes out as Inf or NaN or so small
// that its products may have underflowed, the tile is formed once more by FMAs, as gemm_f32_kernel forms it.
#pragma once
#include "gemm_f32.cuh"
#include "sm100_ptx.cuh"

#include <utility>

namespace alpha {

constexpr int kPlaneThreads = 576, kPlaneBM = 128, kPlaneBK = 32, kPlaneRing = 4;

__host__ __device__ constexpr uint32_t plane_stage_bytes(int BN) { return 3u * (kPlaneBM + BN) * kPlaneBK * 2; }
__host__ __device__ constexpr uint32_t plane_smem_bytes(int BN) { return kPlaneRing * plane_stage_bytes(BN) + 1024; }

__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// x = h + m + l: the planes of four consecutive elements, eight bytes each.  h and m are rounded to nearest.  What the lowest 16 bits of
// `lost` hold afterwards is zero as long as nothing was: an element from 2^-110 on has its last bit at 2^-133 or above, the smallest of bf16;
// of a smaller one, of an Inf and of a NaN there may be a rest.
__device__ __forceinline__ void split_planes(const float4& v, uint2& h, uint2& m, uint2& l, uint32_t& lost)
{
    auto pair = [](float a, float b) {                    // two bf16 words, a in the lower half
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
        return r;
    };
    auto less = [](float a, float b, uint32_t w, float& x, float& y) {   // what a pair leaves of its elements (exact)
        unpack2(sub2(pack2(a, b), pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u))), x, y);
    };
    float r0, r1, r2, r3;
    h = make_uint2(pair(v.x, v.y), pair(v.z, v.w));
    less(v.x, v.y, h.x, r0, r1);
    less(v.z, v.w, h.y, r2, r3);
    m = make_uint2(pair(r0, r1), pair(r2, r3));
    less(r0, r1, m.x, r0, r1);
    less(r2, r3, m.y, r2, r3);
    lost |= __float_as_uint(r0) | __float_as_uint(r1) | __float_as_uint(r2) | __float_as_uint(r3);
    l = make_uint2(__byte_perm(__float_as_uint(r0), __float_as_uint(r1), 0x7632), __byte_perm(__float_as_uint(r2), __float_as_uint(r3), 0x7632));
}

// Zeros past the first n elements.
__device__ __forceinline__ void keep_first(float4& v, int n)
{
    if (n < 2) v.y = 0.f;
    if (n < 3) v.z = 0.f;
    if (n < 4) v.w = 0.f;
}

__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint2 v)
{
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}

// Word i of a thread in a stage of 32 steps x COLS columns: its first column, its first step, its place in a plane.  KC: memory
// runs along k (four steps of one column), else along the columns.
template <int COLS, bool KC> __device__ __forceinline__ int plane_col(int tid, int i)
{
    return KC ? i * 32 + (tid >> 3) : ((tid >> 5) + 8 * i) % (COLS / 32) * 32 + (tid & 7) * 4;
}
template <int COLS, bool KC> __device__ __forceinline__ int plane_k(int tid, int i)
{
    return KC ? (tid & 7) * 4 : ((tid >> 5) + 8 * i) / (COLS / 32) * 4 + ((tid >> 3) & 3);
}
// Place of a thread's first word in a plane, and from one of its words to the next.
template <int COLS, bool KC> __device__ __forceinline__ uint32_t plane_offset(int tid)
{
    const int c = plane_col<COLS, KC>(tid, 0), k = plane_k<COLS, KC>(tid, 0);
    if (KC) return (c >> 3) * 512 + (c & 7) * 64 + (((k >> 3) ^ ((c >> 1) & 3)) << 4) + ((k >> 2) & 1) * 8;
    return (c >> 5) * 2048 + (k >> 3) * 512 + (k & 7) * 64 + ((((c & 31) >> 3) ^ ((k >> 1) & 3)) << 4) + ((c >> 2) & 1) * 8;
}
template <int COLS, bool KC> __device__ constexpr uint32_t plane_step() { return KC ? 2048u : 2048u / (COLS / 32); }
// Steps from one word of a thread to the next where memory runs along the columns.
template <int COLS> __device__ constexpr int plane_dk() { return 32 / (COLS / 32); }

// ---- what is multiplied ---------------------------------------------------------------------------------------
//
// A policy P (by value, in the kernel's parameters) describes both operands and the result:
//   P::kAk, P::kBk     the operand runs along the reduction in memory (else along its rows / columns); words are four floats either way
//   cta()              tile (bx, by, bz): rows from m0, columns from n0, stages [s0, s1) of 32 steps of K in all; false: there is none
//   a_row, a_step      a word of A lies row.at + step.at floats into a_tensor() and is read where use_a() says (a filter tap may miss the
//   b_row, b_step      image, a row, column or step may not exist); the same for B
//   row_out, store     the row of the result, nullptr where there is none; four consecutive outputs of it; columns(): how many there are from n0 on
// Offsets are 32-bit: tensors have fewer than 2^31 elements (planes_fit).

// Tiles of a launch, x fastest, one a CTA; `first` = tile of CTA 0.
struct PlaneGrid { unsigned first; FastDiv by_x, by_y; };

struct PlaneAt { uint32_t at, bits; };

// A row knows which filter rows and columns meet the image from it (bits 0 ... 14 and 16 ... 30), a step names its own; a step past the end
// needs bit 15, which no row has, and a row past the end has none.
constexpr int kPlaneTaps = 15;
constexpr uint32_t kNoStep = 1u << 15;
__device__ __forceinline__ bool plane_meets(const PlaneAt& row, const PlaneAt& step) { return (row.bits & step.bits) == step.bits; }
__device__ __forceinline__ uint32_t tap_bits(unsigned u, unsigned v) { return 1u << u | 0x10000u << v; }

// deltaX of any stride: rows = the pixels of one stride phase (py, px), which all meet the same filter taps, columns = input
// channels, reduction = those taps x output channels (tap-major, without gaps between taps), in `ksplit` parts.  A launch computes
// `parts` of them from part0 on, bz = phase * parts + part, each into its own copy of deltaX, every element of which some phase
// writes; or, without memory for copies, one part that is added to what `out` holds (ADD).
struct PlaneDxProblem {
    static constexpr bool kAk = true, kBk = false, kTail = false, kCopyB = true;
    const float* dY; const float* W; float* out;
    int N, IH, IW, IC, FH, FW, OH, OW, OC, sh, sw, ph, pw;
    int nsw;                       // phases along a row: min(sw, IW)
    int ksplit, parts, part0;
    size_t size;                   // elements of deltaX
    // divisions by OC, and by what phases have one more or less of: A * B, B, Ux (set_divisions)
    FastDiv by_OC, by_AB[4], by_B[2], by_Ux[2];
    int row0[16];                  // first row of each phase among the planes of W
    struct Cta { int m0, n0, s0, s1, K, rows, A, B, py, px, ry, rx, qy, qx, Uy, Ux, row0; FastDiv by_B, by_AB, by_Ux; float* out; };

    void set_divisions()
    {
        const int A = (IH + sh - 1) / sh, B = (IW + sw - 1) / sw, Ux = (FW + sw - 1) / sw;
        auto by = [](int d) { return fast_div(d > 0 ? d : 1); };
        by_OC = by(OC);
        for (int i = 0; i < 4; ++i) by_AB[i] = by((A - i / 2) * (B - i % 2));
        for (int i = 0; i < 2; ++i) { by_B[i] = by(B - i); by_Ux[i] = by(Ux - i); }
    }
    __device__ bool cta(Cta& c, int BM, int BN, int bx, int by, int z) const
    {
        const int phase = z / parts, copy = z - phase * parts, sp = part0 + copy;
        c.py = phase / nsw; c.px = phase - c.py * nsw;
        c.A = (IH - c.py + sh - 1) / sh; c.B = (IW - c.px + sw - 1) / sw;
        c.rows = N * c.A * c.B;
        c.m0 = bx * BM; c.n0 = by * BN;
        if (c.m0 >= c.rows) return false;
        c.ry = (c.py + ph) % sh; c.rx = (c.px + pw) % sw;
        c.qy = (c.py + ph - c.ry) / sh; c.qx = (c.px + pw - c.rx) / sw;
        c.Uy = c.ry < FH ? (FH - c.ry + sh - 1) / sh : 0;
        c.Ux = c.rx < FW ? (FW - c.rx + sw - 1) / sw : 0;
        c.K = c.Uy * c.Ux * OC;
        const int la = c.A * sh < IH ? 1 : 0, lb = c.B * sw < IW ? 1 : 0;                 // a row, a column less than phase 0
        c.by_AB = by_AB[2 * la + lb]; c.by_B = by_B[lb]; c.by_Ux = by_Ux[c.Ux * sw < FW ? 1 : 0];
        c.row0 = row0[phase & 15];
        const int stages = (c.K + 31) / 32, per = (stages + ksplit - 1) / ksplit;
        c.s0 = sp * per < stages ? sp * per : stages;
        c.s1 = c.s0 + per < stages ? c.s0 + per : stages;
        c.out = out + static_cast<size_t>(copy) * size;
        return true;
    }
    __device__ int columns(const Cta& c) const { return IC - c.n0; }
    __device__ const float* a_tensor(const Cta&) const { return dY; }
    __device__ const float* b_tensor(const Cta&) const { return W; }
    // pixel (n, a, b) of the phase
    __device__ bool pixel(const Cta& c, int m, unsigned& n, unsigned& a, unsigned& b) const
    {
        const int r = c.m0 + m;
        if (r >= c.rows) return false;
        unsigned q;
        c.by_AB.divmod(static_cast<unsigned>(r), n, q);
        c.by_B.divmod(q, a, b);
        return true;
    }
    __device__ PlaneAt a_row(const Cta& c, int m) const
    {
        unsigned n, a, b;
        if (!pixel(c, m, n, a, b)) return PlaneAt{0u, 0u};
        const int y = static_cast<int>(a) + c.qy, x = static_cast<int>(b) + c.qx;
        uint32_t taps = 0;
        for (int v = 0; v < c.Ux; ++v)
            if (static_cast<unsigned>(x - v) < static_cast<unsigned>(OW)) taps |= 0x10000u << v;
        for (int u = 0; u < c.Uy; ++u)
            if (static_cast<unsigned>(y - u) < static_cast<unsigned>(OH)) taps |= 1u << u;
        return PlaneAt{static_cast<uint32_t>(((static_cast<int>(n) * OH + y) * OW + x) * OC), taps};
    }
    __device__ void tap(const Cta& c, int k, unsigned& t, unsigned& oc, unsigned& u, unsigned& v) const
    {
        by_OC.divmod(static_cast<unsigned>(k), t, oc);
        c.by_Ux.divmod(t, u, v);
    }
    __device__ PlaneAt a_step(const Cta& c, int k) const
    {
        unsigned t, oc, u, v;
        tap(c, k, t, oc, u, v);
        return PlaneAt{oc - (u * OW + v) * OC, k < c.K ? tap_bits(u, v) : kNoStep};
    }
    __device__ PlaneAt b_row(const Cta& c, int col) const
    {
        return PlaneAt{static_cast<uint32_t>((c.ry * FW + c.rx) * IC + c.n0 + col), c.n0 + col < IC ? 1u : 0u};
    }
    __device__ PlaneAt b_step(const Cta& c, int k) const
    {
        unsigned t, oc, u, v;
        tap(c, k, t, oc, u, v);
        return PlaneAt{(oc * (FH * FW) + u * (sh * FW) + v * sw) * IC, k < c.K ? 1u : kNoStep};
    }
    __device__ static bool use_a(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    __device__ static bool use_b(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    // planes of W with the rows of each phase in the order of its steps: a box of 32 columns x 32 steps x column blocks x planes
    __device__ void copy_b(const Cta& c, uint32_t dst, const CUtensorMap* m, uint32_t bar, int k) const
    {
        tma_load_4d_a(dst, m, bar, 0, c.row0 + k, c.n0 >> 5, 0);
    }
    __device__ float* row_out(const Cta& c, int m) const
    {
        unsigned n, a, b;
        if (!pixel(c, m, n, a, b)) return nullptr;
        return c.out + ((static_cast<size_t>(n) * IH + (a * sh + c.py)) * IW + (b * sw + c.px)) * IC;
    }
};
template <bool ADD>
struct PlaneDx : PlaneDxProblem {
    __device__ void store(const Cta& c, float* row, int col, const float4& o) const
    {
        if (!row || c.n0 + col >= IC) return;
        float4* p = reinterpret_cast<float4*>(row + c.n0 + col);
        if (ADD) {
            const float4 a = *p;
            *p = make_float4(a.x + o.x, a.y + o.y, a.z + o.z, a.w + o.w);
        } else {
            *p = o;
        }
    }
};

// C[b] = A[b] * B[b] over N x M outputs and K steps, with row pitches.  A_KC: A[b] is [N][lda] (else [K][lda], the transposed
// form); B_KC: B[b] is [M][ldb] (else [K][ldb]).  Pitches are multiples of 4 and every matrix starts on a 16-byte boundary;
// words are loaded whole where they start inside the matrix: rows past N and steps past K become zeros (kTail).
template <bool A_KC, bool B_KC>
struct PlaneBatch {
    static constexpr bool kAk = A_KC, kBk = B_KC, kTail = true, kCopyB = false;
    const float *A, *B; float* C;
    int N, M, K, lda, ldb, ldc;
    size_t strA, strB, strC;
    struct Cta { int m0, n0, s0, s1, K; const float *A, *B; float* C; };

    __device__ bool cta(Cta& c, int BM, int BN, int bx, int by, int bz) const
    {
        c.m0 = by * BM; c.n0 = bx * BN;
        c.s0 = 0; c.s1 = (K + 31) / 32; c.K = K;
        c.A = A + static_cast<size_t>(bz) * strA; c.B = B + static_cast<size_t>(bz) * strB; c.C = C + static_cast<size_t>(bz) * strC;
        return true;
    }
    __device__ int columns(const Cta& c) const { return M - c.n0; }
    // rows from one of the tile to the end of the matrix (the columns of a B that runs along them are a multiple of 4)
    __device__ int a_left(const Cta& c, int m) const { return N - (c.m0 + m); }
    __device__ const float* a_tensor(const Cta& c) const { return c.A; }
    __device__ const float* b_tensor(const Cta& c) const { return c.B; }
    __device__ PlaneAt a_row(const Cta& c, int m) const { return PlaneAt{static_cast<uint32_t>((c.m0 + m) * (A_KC ? lda : 1)), c.m0 + m < N ? 1u : 0u}; }
    __device__ PlaneAt b_row(const Cta& c, int col) const { return PlaneAt{static_cast<uint32_t>((c.n0 + col) * (B_KC ? ldb : 1)), c.n0 + col < M ? 1u : 0u}; }
    __device__ PlaneAt a_step(const Cta&, int k) const { return PlaneAt{static_cast<uint32_t>(k * (A_KC ? 1 : lda)), k < K ? 1u : kNoStep}; }
    __device__ PlaneAt b_step(const Cta&, int k) const { return PlaneAt{static_cast<uint32_t>(k * (B_KC ? 1 : ldb)), k < K ? 1u : kNoStep}; }
    __device__ static bool use_a(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    __device__ static bool use_b(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    __device__ float* row_out(const Cta& c, int m) const { return c.m0 + m < N ? c.C + static_cast<size_t>(c.m0 + m) * ldc : nullptr; }
    __device__ void store(const Cta& c, float* row, int col, const float4& o) const
    {
        const int j = c.n0 + col;
        if (!row || j >= M) return;
        if (j + 3 < M) { *reinterpret_cast<float4*>(row + j) = o; return; }
        row[j] = o.x;
        if (j + 1 < M) row[j + 1] = o.y;
        if (j + 2 < M) row[j + 2] = o.z;
    }
};

// Forward convolution: rows = output pixels, columns = output channels, reduction = taps x input channels, as a row of W holds them.
// bz = part of the reduction, each into its own copy of Y (bias and activation only without parts).
struct PlaneFwd {
    static constexpr bool kAk = true, kBk = true, kTail = false, kCopyB = true;
    const float* X; const float* W; const float* bias; float* out;
    int N, IH, IW, IC, FH, FW, OH, OW, OC, sh, sw, ph, pw, K, rows, ksplit, act_on;
    float act_k;
    size_t size;                   // elements of Y
    FastDiv by_OW, by_OHW, by_IC, by_FW;
    struct Cta { int m0, n0, s0, s1, K; float* out; };

    __device__ bool cta(Cta& c, int BM, int BN, int bx, int by, int sp) const
    {
        c.m0 = bx * BM; c.n0 = by * BN;
        const int stages = (K + 31) / 32, per = (stages + ksplit - 1) / ksplit;
        c.s0 = sp * per < stages ? sp * per : stages;
        c.s1 = c.s0 + per < stages ? c.s0 + per : stages;
        c.K = K;
        c.out = out + static_cast<size_t>(sp) * size;
        return true;
    }
    __device__ int columns(const Cta& c) const { return OC - c.n0; }
    __device__ const float* a_tensor(const Cta&) const { return X; }
    __device__ const float* b_tensor(const Cta&) const { return W; }
    __device__ PlaneAt a_row(const Cta& c, int m) const
    {
        if (c.m0 + m >= rows) return PlaneAt{0u, 0u};
        unsigned n, q, oh, ow;
        by_OHW.divmod(static_cast<unsigned>(c.m0 + m), n, q);
        by_OW.divmod(q, oh, ow);
        const int y = static_cast<int>(oh) * sh - ph, x = static_cast<int>(ow) * sw - pw;
        uint32_t taps = 0;
        for (int v = 0; v < FW; ++v)
            if (static_cast<unsigned>(x + v) < static_cast<unsigned>(IW)) taps |= 0x10000u << v;
        for (int u = 0; u < FH; ++u)
            if (static_cast<unsigned>(y + u) < static_cast<unsigned>(IH)) taps |= 1u << u;
        return PlaneAt{static_cast<uint32_t>(((static_cast<int>(n) * IH + y) * IW + x) * IC), taps};
    }
    __device__ PlaneAt a_step(const Cta&, int k) const
    {
        unsigned t, ic, fh, fw;
        by_IC.divmod(static_cast<unsigned>(k), t, ic);
        by_FW.divmod(t, fh, fw);
        return PlaneAt{(fh * IW + fw) * IC + ic, k < K ? tap_bits(fh, fw) : kNoStep};
    }
    __device__ PlaneAt b_row(const Cta& c, int col) const { return PlaneAt{static_cast<uint32_t>((c.n0 + col) * K), c.n0 + col < OC ? 1u : 0u}; }
    __device__ PlaneAt b_step(const Cta&, int k) const { return PlaneAt{static_cast<uint32_t>(k), k < K ? 1u : kNoStep}; }
    __device__ static bool use_a(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    __device__ static bool use_b(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    // planes of W, rows padded to whole stages: a box of 32 steps x BN rows x planes
    __device__ void copy_b(const Cta& c, uint32_t dst, const CUtensorMap* m, uint32_t bar, int k) const { tma_load_3d_a(dst, m, bar, k, c.n0, 0); }
    __device__ float* row_out(const Cta& c, int m) const { return c.m0 + m < rows ? c.out + static_cast<size_t>(c.m0 + m) * OC : nullptr; }
    __device__ void store(const Cta& c, float* row, int col, float4 o) const
    {
        const int j = c.n0 + col;
        if (!row || j >= OC) return;
        if (bias) {
            const float4 b = *reinterpret_cast<const float4*>(bias + j);
            o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
        }
        if (act_on) {
            o.x = o.x > 0.f ? o.x : act_k * o.x; o.y = o.y > 0.f ? o.y : act_k * o.y;
            o.z = o.z > 0.f ? o.z : act_k * o.z; o.w = o.w > 0.f ? o.w : act_k * o.w;
        }
        *reinterpret_cast<float4*>(row + j) = o;
    }
};

// deltaW: rows = output channels, columns = taps x input channels, reduction = output pixels, in parts like PlaneFwd.
struct PlaneDw {
    static constexpr bool kAk = false, kBk = false, kTail = false, kCopyB = false;
    const float* dY; const float* X; float* out;
    int IH, IW, IC, FW, OC, sh, sw, ph, pw, K, L, ksplit;    // K pixels, L = taps * IC floats of a row of deltaW
    size_t size;
    FastDiv by_OW, by_OHW, by_IC, by_FW;
    struct Cta { int m0, n0, s0, s1, K; float* out; };
    static constexpr int kNone = 1 << 30;                   // as fh: no such column, as y: no such step (added without sign: 2^31 is no row either)
    struct BRow { uint32_t at; int fh, fw; };
    struct BStep { uint32_t at; int y, x; };

    __device__ bool cta(Cta& c, int BM, int BN, int bx, int by, int sp) const
    {
        c.m0 = bx * BM; c.n0 = by * BN;
        const int stages = (K + 31) / 32, per = (stages + ksplit - 1) / ksplit;
        c.s0 = sp * per < stages ? sp * per : stages;
        c.s1 = c.s0 + per < stages ? c.s0 + per : stages;
        c.K = K;
        c.out = out + static_cast<size_t>(sp) * size;
        return true;
    }
    __device__ int columns(const Cta& c) const { return L - c.n0; }
    __device__ const float* a_tensor(const Cta&) const { return dY; }
    __device__ const float* b_tensor(const Cta&) const { return X; }
    __device__ PlaneAt a_row(const Cta& c, int m) const { return PlaneAt{static_cast<uint32_t>(c.m0 + m), c.m0 + m < OC ? 1u : 0u}; }
    __device__ PlaneAt a_step(const Cta&, int k) const { return PlaneAt{static_cast<uint32_t>(k * OC), k < K ? 1u : kNoStep}; }
    __device__ BRow b_row(const Cta& c, int col) const
    {
        const int q = c.n0 + col;
        if (q >= L) return BRow{0u, kNone, 0};
        unsigned t, ic, fh, fw;
        by_IC.divmod(static_cast<unsigned>(q), t, ic);
        by_FW.divmod(t, fh, fw);
        return BRow{(fh * IW + fw) * IC + ic, static_cast<int>(fh), static_cast<int>(fw)};
    }
    __device__ BStep b_step(const Cta&, int k) const
    {
        unsigned n, q, oh, ow;
        by_OHW.divmod(static_cast<unsigned>(k), n, q);
        by_OW.divmod(q, oh, ow);
        const int y = static_cast<int>(oh) * sh - ph, x = static_cast<int>(ow) * sw - pw;
        return BStep{static_cast<uint32_t>(((static_cast<int>(n) * IH + y) * IW + x) * IC), k < K ? y : kNone, x};
    }
    __device__ static bool use_a(const PlaneAt& row, const PlaneAt& step) { return plane_meets(row, step); }
    __host__ __device__ bool use_b(const BRow& row, const BStep& step) const
    {
        return static_cast<unsigned>(step.y) + static_cast<unsigned>(row.fh) < static_cast<unsigned>(IH) && static_cast<unsigned>(step.x + row.fw) < static_cast<unsigned>(IW);
    }
    __device__ float* row_out(const Cta& c, int m) const { return c.m0 + m < OC ? c.out + static_cast<size_t>(c.m0 + m) * L : nullptr; }
    __device__ void store(const Cta& c, float* row, int col, const float4& o) const
    {
        if (row && c.n0 + col < L) *reinterpret_cast<float4*>(row + c.n0 + col) = o;
    }
};

// The 16-byte word `at` floats into a tensor, zeros without `use`: one predicated load, so that a thread's loads leave back to back
// (behind a branch the compiler moves each result to its place before the next load: 240 clocks a word).
__device__ __forceinline__ float4 load_word(const float* tensor, uint32_t at, bool use)
{
    float4 v;
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b64 a;\n\tsetp.ne.u32 q, %6, 0;\n\tmad.wide.u32 a, %5, 4, %4;\n\t"
        "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
        "@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
        : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w) : "l"(tensor), "r"(at), "r"(static_cast<uint32_t>(use)));
    return v;
}

// ---- tiles whose operands or sums the planes do not hold -------------------------------------------------------
//
// The 512 threads that staged the tile form it by FMAs in ascending k, 8 x 4 (4 x 4) outputs each, from words staged in shared memory as they
// are; or, where only bits below 2^-133 were lost (tiny operands beside ordinary ones, as a softmax has them), look at the operands
// once more and let the sums stand.  us, ordinary data / an Inf in every picture / data times 1e-30: 50 x 35 x 29, 36 -> 100 channels 3x3
// forward 34 / 138 / 185, 512 x 8x8 x 128 51 / 489 / 389, 256 x 16x16, 128 -> 256, 4x4 s2 81 / 740 / 695 (a thread per eight rows that read both operands
// from global memory and computed their places anew for every step: 2019 / 5862, 12749, 22740; data times 1e-25 as well, which now stays);
// a softmax with tails, 64 x 130 x 200 x 130, 45 where ordinary data take 32 and the FMA kernel 40.

// Barrier of those threads; whether any of them says so.
__device__ __forceinline__ bool again_or(bool x)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 512, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(static_cast<uint32_t>(x)) : "memory");
    return r != 0;
}

template <int BN, class P>
struct PlaneAgain {
    using ARow = decltype(std::declval<const P&>().a_row(std::declval<const typename P::Cta&>(), 0));
    using BRow = decltype(std::declval<const P&>().b_row(std::declval<const typename P::Cta&>(), 0));
    using AStep = decltype(std::declval<const P&>().a_step(std::declval<const typename P::Cta&>(), 0));
    using BStep = decltype(std::declval<const P&>().b_step(std::declval<const typename P::Cta&>(), 0));
    struct Shared {
        float a[2][32][kPlaneBM + 4], b[2][32][BN + 4];      // [stage & 1][step][row or column]
        AStep sa[32];
        BStep sb[32];
        uint32_t any_a[kPlaneBM], any_b[BN], top;              // bits set in a row of A, a column of B; the largest word
    };
    static_assert(sizeof(Shared) % 4 == 0 && sizeof(Shared) + 512 * BN <= kPlaneRing * plane_stage_bytes(BN), "shared memory");
    static constexpr int TM = BN / 16, CG = BN / 4, NB = BN / 64;

    // The words of a stage that a thread loads: two of A, NB of B.
    const P& p;
    const typename P::Cta& c;
    const ARow* rows;
    int tid;
    const float *A, *B;
    float4 va[2], vb[NB];
    __device__ PlaneAgain(const P& p_, const typename P::Cta& c_, const ARow* rows_, int tid_) : p(p_), c(c_), rows(rows_), tid(tid_), A(p_.a_tensor(c_)), B(p_.b_tensor(c_)) {}
    __device__ int a_col(int i) const { return P::kAk ? (tid >> 3) + 64 * i : (tid & 31) * 4; }
    __device__ int a_k(int i) const { return P::kAk ? (tid & 7) * 4 : (tid >> 5) + 16 * i; }
    __device__ int b_col(int i) const { return P::kBk ? (tid >> 3) + 64 * i : tid % CG * 4; }
    __device__ int b_k(int i) const { return P::kBk ? (tid & 7) * 4 : tid / CG + 512 / CG * i; }
    __device__ ARow a_row(int m) const
    {
        if constexpr (P::kAk) return rows[m];
        else return p.a_row(c, m);
    }
    __device__ void load(int s)
    {
        const int k0 = (c.s0 + s) * 32;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const ARow r = a_row(a_col(i));
            const AStep at = p.a_step(c, k0 + a_k(i));
            va[i] = load_word(A, r.at + at.at, p.use_a(r, at));
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const BRow r = p.b_row(c, b_col(i));
            const BStep at = p.b_step(c, k0 + b_k(i));
            vb[i] = load_word(B, r.at + at.at, p.use_b(r, at));
        }
    }
    __device__ static uint32_t top_of(const float4& v)
    {
        const uint32_t a = __float_as_uint(v.x) & 0x7fffffffu, b = __float_as_uint(v.y) & 0x7fffffffu, d = __float_as_uint(v.z) & 0x7fffffffu, e = __float_as_uint(v.w) & 0x7fffffffu;
        return max(max(a, b), max(d, e));
    }
    __device__ uint32_t top() const
    {
        uint32_t t = max(top_of(va[0]), top_of(va[1]));
#pragma unroll
        for (int i = 0; i < NB; ++i) t = max(t, top_of(vb[i]));
        return t;
    }
    // Joins the bits of N words into those of their rows (columns): four of a word, or, where it runs along k, one.
    template <bool K_MAJOR, int N>
    __device__ static void join(const float4 (&v)[N], uint32_t (&bits)[4])
    {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t x = __float_as_uint(v[i].x) << 1, y = __float_as_uint(v[i].y) << 1, z = __float_as_uint(v[i].z) << 1, w = __float_as_uint(v[i].w) << 1;
            if (K_MAJOR) bits[i] |= x | y | z | w;
            else { bits[0] |= x; bits[1] |= y; bits[2] |= z; bits[3] |= w; }
        }
    }
    template <bool K_MAJOR, int PITCH>
    __device__ static void put(float (*to)[PITCH], int k, int col, const float4& v)
    {
        if (K_MAJOR) { to[k][col] = v.x; to[k + 1][col] = v.y; to[k + 2][col] = v.z; to[k + 3][col] = v.w; }
        else *reinterpret_cast<float4*>(&to[k][col]) = v;
    }
    // Steps [0, n) of a staged stage.  MASKED: a product whose tap misses the image, or with no operand at all, is left out, so that an Inf
    // or NaN of the other operand stays out of it (among finite words the zeros in their place do the same).
    template <bool MASKED>
    __device__ void add(const Shared& m, int buf, int n, int row, int col, float (&acc)[TM][4]) const
    {
        BRow rb{};
        if (MASKED) rb = p.b_row(c, col);
#pragma unroll 2
        for (int k = 0; k < n; ++k) {
            const float4 b = *reinterpret_cast<const float4*>(&m.b[buf][k][col]);
            float a[TM];
#pragma unroll
            for (int y = 0; y < TM; y += 4) *reinterpret_cast<float4*>(a + y) = *reinterpret_cast<const float4*>(&m.a[buf][k][row + y]);
            if (MASKED && !p.use_b(rb, m.sb[k])) continue;
#pragma unroll
            for (int y = 0; y < TM; ++y) {
                if (MASKED && !p.use_a(a_row(P::kAk ? row + y : (row + y) & ~3), m.sa[k])) continue;
                acc[y][0] = fmaf(a[y], b.x, acc[y][0]); acc[y][1] = fmaf(a[y], b.y, acc[y][1]);
                acc[y][2] = fmaf(a[y], b.z, acc[y][2]); acc[y][3] = fmaf(a[y], b.w, acc[y][3]);
            }
        }
    }
};

template <int BN, class P>
__device__ __forceinline__ void gemm_planes_again(const P& p, const typename P::Cta& c, const typename PlaneAgain<BN, P>::ARow* rows, float* const* outs, uint8_t* smem, int tid)
{
    using G = PlaneAgain<BN, P>;
    typename G::Shared& m = *reinterpret_cast<typename G::Shared*>(smem);
    G g(p, c, rows, tid);
    const int col = tid % G::CG * 4, row = tid / G::CG * G::TM, stages = c.s1 - c.s0;
    float acc[G::TM][4] = {};
    g.load(0);
    for (int s = 0; s < stages; ++s) {
        const int buf = s & 1, k0 = (c.s0 + s) * 32, n = c.K - k0 < 32 ? c.K - k0 : 32;
#pragma unroll
        for (int i = 0; i < 2; ++i) G::template put<P::kAk>(m.a[buf], g.a_k(i), g.a_col(i), g.va[i]);
#pragma unroll
        for (int i = 0; i < G::NB; ++i) G::template put<P::kBk>(m.b[buf], g.b_k(i), g.b_col(i), g.vb[i]);
        const bool masked = again_or(g.top() >= 0x7f800000u);       // (the other buffer may still be read, this one no more)
        if (s + 1 < stages) g.load(s + 1);
        if (masked) {
            // (a step of an operand that runs along k is known by its word of four)
            if (tid < 32) m.sa[tid] = p.a_step(c, k0 + (P::kAk ? tid & ~3 : tid));
            else if (tid < 64) m.sb[tid - 32] = p.b_step(c, k0 + (P::kBk ? tid - 32 & ~3 : tid - 32));
            again_or(false);
            g.template add<true>(m, buf, n, row, col, acc);
        } else {
            g.template add<false>(m, buf, n, row, col, acc);
        }
    }
#pragma unroll
    for (int y = 0; y < G::TM; ++y) p.store(c, outs[row + y], col, make_float4(acc[y][0], acc[y][1], acc[y][2], acc[y][3]));
}

// Whether the sums of a thread, column x at sums[512 x], x < end, of a row stand although operands lost bits: less than 2^-133 of one, times its
// partner, for each of two operands and every step, is less than 2^-24 of a sum.  (A zero column, as a padded matrix has, gives zeros.)
template <int BN, class P>
__device__ __forceinline__ bool planes_suffice(const P& p, const typename P::Cta& c, const typename PlaneAgain<BN, P>::ARow* rows, uint8_t* smem, int tid, const float* sums,
                                               int row, int col0, int end)
{
    using G = PlaneAgain<BN, P>;
    typename G::Shared& m = *reinterpret_cast<typename G::Shared*>(smem);
    G g(p, c, rows, tid);
    if (tid < kPlaneBM) m.any_a[tid] = 0;
    if (tid < BN) m.any_b[tid] = 0;
    if (tid == 0) m.top = 0;
    uint32_t top = 0, any_a[4] = {}, any_b[4] = {};
    for (int s = 0; s < c.s1 - c.s0; ++s) {
        g.load(s);
        top = max(top, g.top());
        G::template join<P::kAk>(g.va, any_a);
        G::template join<P::kBk>(g.vb, any_b);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    again_or(false);
    if ((tid & 31) == 0) atomicMax(&m.top, top);
#pragma unroll
    for (int i = 0; i < (P::kAk ? 2 : 4); ++i) atomicOr(&m.any_a[P::kAk ? g.a_col(i) : g.a_col(0) + i], any_a[i]);
#pragma unroll
    for (int i = 0; i < (P::kBk ? G::NB : 4); ++i) atomicOr(&m.any_b[P::kBk ? g.b_col(i) : g.b_col(0) + i], any_b[i]);
    again_or(false);
    const float least = __uint_as_float(m.top) * static_cast<float>((c.s1 - c.s0) * 64) * 0x1p-109f;
    bool stand = true;
    if (m.any_a[row])
        for (int x = 0; x < BN / 4 && x < end; ++x)
            if (!(fabsf(sums[x * 512]) >= least) && m.any_b[col0 + x]) stand = false;
    return !again_or(!stand);
}

// What becomes of a tile some thread of which found operands that lost bits or (`again`) sums that the planes may not have formed.  The sums lie
// behind Shared, BN / 4 columns of a row a thread (a call of its own, so that the kernel's registers need not outlive one).
template <int BN, class P>
__device__ __noinline__ void gemm_planes_look(const P& p, const typename P::Cta& c, const typename PlaneAgain<BN, P>::ARow* rows, float* const* outs, uint8_t* smem, int tid, bool again)
{
    constexpr int COLS = BN / 4;
    again = again_or(again);
    if (!again) {
        const float* sums = reinterpret_cast<const float*>(smem + sizeof(typename PlaneAgain<BN, P>::Shared)) + tid;
        const int row = ((tid >> 5) & 3) * 32 + (tid & 31);
        float* out = outs[row];
        const int col0 = (tid >> 7) * COLS, end = (out ? p.columns(c) : 0) - col0;
        again = !planes_suffice<BN>(p, c, rows, smem, tid, sums, row, col0, end);
        if (!again)
            for (int x = 0; x < COLS; x += 4) p.store(c, out, col0 + x, make_float4(sums[x * 512], sums[x * 512 + 512], sums[x * 512 + 1024], sums[x * 512 + 1536]));
    }
    if (again) gemm_planes_again<BN>(p, c, rows, outs, smem, tid);
}

// After a wait that ran out: time for what has been issued to end, before shared and tensor memory are given back.
static __device__ __noinline__ void settle()
{
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) {}
}

template <int BN, class P, bool TMA_B>
__global__ void __launch_bounds__(kPlaneThreads, 1) gemm_planes_kernel(const __grid_constant__ P p, const __grid_constant__ CUtensorMap tmB, const PlaneGrid grid, int* status)
{
    static_assert(BN == 64 || BN == 128, "tile shape");
    constexpr int NA = kPlaneBM / 32, NB = BN / 32, COLS = BN / 4;      // words of a thread in a stage; columns of a warp
    constexpr uint32_t kPlaneA = kPlaneBM * kPlaneBK * 2, kPlaneB = BN * kPlaneBK * 2, kStage = plane_stage_bytes(BN), kTmem = BN == 64 ? 256 : 512;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bars[2 * kPlaneRing + 2];
    __shared__ uint32_t tmem_holder;
    __shared__ typename P::Cta c;                            // (in registers or local memory it would cost the loops)
    __shared__ int work;
    __shared__ decltype(p.a_row(c, 0)) rows[P::kAk ? kPlaneBM : 1];   // computed once: 16 threads read a row, and divisions cost
    __shared__ float* outs[kPlaneBM];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full_a = smem_u32(bars), done_a = full_a + 8 * kPlaneRing, free_a = done_a + 8 * kPlaneRing;
    if (tid == 0) {
        for (int i = 0; i < kPlaneRing; ++i) {
            mbar_init(&bars[i], TMA_B ? 9 : 8);          // a stage is staged: one arrival per warp of its group, one for the copy of B
            mbar_init(&bars[kPlaneRing + i], 1);         // its MMAs are done
        }
        mbar_init(&bars[2 * kPlaneRing], 16);            // an hh accumulator has been read by all warps
        mbar_init(&bars[2 * kPlaneRing + 1], 16);
        fence_barrier_init();
        typename P::Cta mine;
        unsigned bx, by, bz, q;
        grid.by_x.divmod(grid.first + blockIdx.x, q, bx);
        grid.by_y.divmod(q, bz, by);
        work = p.cta(mine, kPlaneBM, BN, static_cast<int>(bx), static_cast<int>(by), static_cast<int>(bz));
        c = mine;
    }
    if (warp == 16) {
        tmem_alloc(&tmem_holder, kTmem);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_holder;

    const int stages = work && c.s1 > c.s0 ? c.s1 - c.s0 : 0;
    if (work) {
        if (P::kAk && tid < kPlaneBM) rows[tid] = p.a_row(c, tid);
        else if (tid >= kPlaneBM && tid < 2 * kPlaneBM) outs[tid - kPlaneBM] = p.row_out(c, tid - kPlaneBM);
    }
    __syncthreads();
    bool ok = true, again = false, look = false;
    unsigned long long acc[COLS / 2];
#pragma unroll
    for (int x = 0; x < COLS / 2; ++x) acc[x] = 0ull;
    // tensor memory: [hh of even windows][hm + mh][hl + mm + lh][hh of odd windows]
    constexpr uint32_t kSide = BN, kOdd = 3 * BN;

    if (warp == 17) {
        grid_dependency_wait();
        grid_dependency_trigger();
        if constexpr (TMA_B) if (elect_one()) {
            for (int s = 0; s < stages; ++s) {
                const uint32_t slot = s % kPlaneRing, bar = full_a + 8 * slot;
                if (s >= kPlaneRing && !mbar_wait_a(done_a + 8 * slot, (s / kPlaneRing - 1) & 1)) { report(status, kStatusProducerTimeout); settle(); break; }
                mbar_arrive_expect_tx_a(bar, 3 * kPlaneB);
                p.copy_b(c, smem_u32(smem) + slot * kStage + 3 * kPlaneA, &tmB, bar, (c.s0 + s) * 32);
            }
        }
        __syncwarp();
    } else if (warp == 16) {
        grid_dependency_wait();
        grid_dependency_trigger();
        // The whole warp walks the stages, so that counters and descriptors are uniform values; one lane issues.
        constexpr uint32_t dhi = (512u >> 4) | (1u << 14) | (static_cast<uint32_t>(kSwizzle64B) << 29);
        constexpr uint32_t a_k = P::kAk ? 2u : 64u, b_k = P::kBk ? 2u : 64u;          // 16 steps further, in 16-byte units
        constexpr uint32_t i1 = make_idesc_bf16(128, BN, !P::kAk, !P::kBk), i2 = make_idesc_bf16(128, 2 * BN, !P::kAk, !P::kBk),
                           i3 = make_idesc_bf16(128, BN == 64 ? 192 : 128, !P::kAk, !P::kBk);
        constexpr uint32_t pa = kPlaneA >> 4, pb = kPlaneB >> 4;
        const uint32_t base = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint32_t a_lo0 = smem_desc_lo(base, P::kAk ? 16u : 2048u), b_lo0 = smem_desc_lo(base + 3 * kPlaneA, P::kBk ? 16u : 2048u);
        const uint32_t side = tmem + kSide, elected = elect_one();
        const int left = c.K - c.s0 * 32;                                            // steps from the first stage on
        for (int s = 0; s < stages; ++s) {
            const uint32_t slot = s % kPlaneRing, window = s >> 1, d = tmem + (window & 1 ? kOdd : 0u);
            ok = mbar_wait_a(full_a + 8 * slot, (s / kPlaneRing) & 1);
            if (ok && !(s & 1) && window >= 2) ok = mbar_wait_a(free_a + 8 * (window & 1), ((window >> 1) - 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) { report(status, kStatusMmaTimeout); settle(); break; }
            tc_fence_after_sync();
            const uint32_t a = a_lo0 + slot * (kStage >> 4), b = b_lo0 + slot * (kStage >> 4);
            const uint32_t keep = s & 1, keep_side = s ? 1u : 0u;
            auto step = [&](auto k_, uint32_t keep, uint32_t keep_side) {
                constexpr uint32_t ka = decltype(k_)::value * a_k, kb = decltype(k_)::value * b_k;
                // columns: [hh][hm + mh][hl + mm + lh]
                if (BN == 64 && keep && !(window & 1)) {
                    mma_bf16_elected<ka, kb>(d, a, dhi, b, dhi, i3, 1u, elected);
                } else {
                    mma_bf16_elected<ka, kb>(d, a, dhi, b, dhi, i1, keep, elected);
                    mma_bf16_elected<ka, kb + pb>(side, a, dhi, b, dhi, i2, keep_side, elected);
                }
                mma_bf16_elected<ka + pa, kb>(side, a, dhi, b, dhi, i2, 1u, elected);
                mma_bf16_elected<ka + 2 * pa, kb>(side + BN, a, dhi, b, dhi, i1, 1u, elected);
            };
            step(std::integral_constant<uint32_t, 0>{}, keep, keep_side);
            if (left - s * 32 > 16) step(std::integral_constant<uint32_t, 1>{}, 1u, 1u);
            if (elected) mma_commit_a(done_a + 8 * slot);
        }
        __syncwarp();
    } else {
        if (!stages) {
            grid_dependency_wait();
            grid_dependency_trigger();
        } else {
        const int group = warp >> 3, t = tid & 255;          // two groups of 256 threads take alternate stages
        // along k a thread's words lie in NA (NB) rows and at one step, else in one column block and plane_dk steps apart
        decltype(p.a_row(c, 0)) ra[P::kAk ? NA : 1];
        decltype(p.b_row(c, 0)) rb[P::kBk && !TMA_B ? NB : 1];
#pragma unroll
        for (int i = 0; i < (P::kAk ? NA : 1); ++i) {
            if constexpr (P::kAk) ra[i] = rows[plane_col<kPlaneBM, true>(t, i)];
            else ra[i] = p.a_row(c, plane_col<kPlaneBM, false>(t, i));
        }
        if constexpr (!TMA_B)
#pragma unroll
            for (int i = 0; i < (P::kBk ? NB : 1); ++i) rb[i] = p.b_row(c, plane_col<BN, P::kBk>(t, i));
        const uint32_t off_a = smem_u32(smem) + plane_offset<kPlaneBM, P::kAk>(t), off_b = smem_u32(smem) + 3 * kPlaneA + plane_offset<BN, P::kBk>(t);
        const float *A = p.a_tensor(c), *B = p.b_tensor(c);
        float4 va[NA], vb[NB];
        uint32_t lost = 0;
        auto load = [&](int s) {
            const int k0 = (c.s0 + s) * 32, ka = k0 + plane_k<kPlaneBM, P::kAk>(t, 0), kb = k0 + plane_k<BN, P::kBk>(t, 0);
            if constexpr (P::kAk) {
                const auto at = p.a_step(c, ka);
#pragma unroll
                for (int i = 0; i < NA; ++i) va[i] = load_word(A, ra[i].at + at.at, p.use_a(ra[i], at));
            } else {
#pragma unroll
                for (int i = 0; i < NA; ++i) {
                    const auto at = p.a_step(c, ka + i * plane_dk<kPlaneBM>());
                    va[i] = load_word(A, ra[0].at + at.at, p.use_a(ra[0], at));
                }
            }
            if constexpr (TMA_B) {
            } else if constexpr (P::kBk) {
                const auto at = p.b_step(c, kb);
#pragma unroll
                for (int i = 0; i < NB; ++i) vb[i] = load_word(B, rb[i].at + at.at, p.use_b(rb[i], at));
            } else {
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    const auto at = p.b_step(c, kb + i * plane_dk<BN>());
                    vb[i] = load_word(B, rb[0].at + at.at, p.use_b(rb[0], at));
                }
            }
        };
        const uint32_t lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (warp >> 2) * COLS;
        // acc += the warp's columns of a column block
        auto add_columns = [&](uint32_t from) {
            // (eight at a time where the words of both operands are in registers too)
            constexpr int C = TMA_B || COLS == 16 ? 16 : 8;
#pragma unroll
            for (int x = 0; x < COLS; x += C) {
                uint32_t v[C];
                if constexpr (C == 16) tmem_ld_32x16(lanes + from + x, v);
                else tmem_ld_32x8(lanes + from + x, v);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < C; q += 2) acc[(x + q) / 2] = add2(acc[(x + q) / 2], pack2(__uint_as_float(v[q]), __uint_as_float(v[q + 1])));
            }
        };
        auto wait_done = [&](int s) {
            ok = __all_sync(0xffffffffu, ok && mbar_wait_a(done_a + 8 * (s % kPlaneRing), (s / kPlaneRing) & 1));
            if (!ok) report(status, kStatusEpilogueTimeout);
            return ok;
        };
        // the hh sum of window w into the running sums
        auto flush = [&](int w) {
            if (!wait_done(2 * w + 1 < stages ? 2 * w + 1 : stages - 1)) return false;
            tc_fence_after_sync();
            add_columns(w & 1 ? kOdd : 0u);
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_a(free_a + 8 * (w & 1));
            return true;
        };
        int flushed = 0;
        grid_dependency_wait();
        grid_dependency_trigger();
        if (group < stages) load(group);
        for (int s = group; s < stages; s += 2) {
            // two windows back: its MMAs are done, or nearly
            if (s >= 4 && !flush(flushed++)) break;
            if (s >= kPlaneRing && !wait_done(s - kPlaneRing)) break;
            const uint32_t at_a = off_a + (s % kPlaneRing) * kStage, at_b = off_b + (s % kPlaneRing) * kStage;
            if constexpr (P::kTail) {
                if constexpr (!P::kAk) {
                    const int left = p.a_left(c, plane_col<kPlaneBM, false>(t, 0));
                    if (left < 4)
#pragma unroll
                        for (int i = 0; i < NA; ++i) keep_first(va[i], left);
                }
                const int steps = c.K - (c.s0 + s) * 32;
                if (steps < 32) {
                    if (P::kAk)
#pragma unroll
                        for (int i = 0; i < NA; ++i) keep_first(va[i], steps - plane_k<kPlaneBM, true>(t, i));
                    if (P::kBk && !TMA_B)
#pragma unroll
                        for (int i = 0; i < NB; ++i) keep_first(vb[i], steps - plane_k<BN, true>(t, i));
                }
            }
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                uint2 h, m, l;
                split_planes(va[i], h, m, l, lost);
                const uint32_t at = at_a + i * plane_step<kPlaneBM, P::kAk>();
                st_shared_v2(at, h); st_shared_v2(at + kPlaneA, m); st_shared_v2(at + 2 * kPlaneA, l);
            }
            if constexpr (!TMA_B)
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                uint2 h, m, l;
                split_planes(vb[i], h, m, l, lost);
                const uint32_t at = at_b + i * plane_step<BN, P::kBk>();
                st_shared_v2(at, h); st_shared_v2(at + kPlaneB, m); st_shared_v2(at + 2 * kPlaneB, l);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_a(full_a + 8 * (s % kPlaneRing));
            // (not before the fence, which waits for loads in flight)
            if (s + 2 < stages) load(s + 2);
        }
        const int windows = (stages + 1) >> 1;
        while (ok && flushed < windows) flush(flushed++);
        if (ok) {
            tc_fence_after_sync();
            add_columns(kSide);
            add_columns(kSide + BN);
            // sums that the planes may not have formed: not finite, or below 2^-110 and not zero, where underflow of 2^-149 a product counts
            // (measured: sums of 2^-124 err by 2e-7, below that by one such unit a product)
            uint32_t most = 0, least = 0xffffffffu;
#pragma unroll
            for (int x = 0; x < COLS / 2; ++x) {
                float a, b;
                unpack2(acc[x], a, b);
                const uint32_t u = __float_as_uint(a) << 1, v = __float_as_uint(b) << 1;
                most = max(most, max(u, v));
                least = min(least, min(u - 1, v - 1));          // (zero as the largest)
            }
            again = most >= 0xff000000u || least < 2u * 0x08800000u;
            // (and a word that is not the sum of its planes: its partner may be so large that the sum does not show it, 1e-37 x 1e11 would
            // err by 6.6e-4)
            look = again || (lost & 0xffffu) != 0;
        }
        }
        tc_fence_before_sync();
    }
    look = __syncthreads_or(look) != 0;       // every MMA has completed: shared memory is free
    if (warp == 16) tmem_dealloc(tmem_base, kTmem);
    if (!work || warp >= 16) return;
    if (look) {
        float* sums = reinterpret_cast<float*>(smem + sizeof(typename PlaneAgain<BN, P>::Shared)) + tid;
#pragma unroll
        for (int x = 0; x < COLS / 2; ++x) unpack2(acc[x], sums[x * 1024], sums[x * 1024 + 512]);
        gemm_planes_look<BN>(p, c, rows, outs, smem, tid, again);
        return;
    }
    if (!ok) return;
    // A lane holds a row; written from the registers, an instruction would touch 32 rows for 16 bytes each.  The warp's block of 32
    // columns goes through 4 KB of shared memory and leaves as whole 128-byte pieces, four rows per instruction.
    const int row0 = (warp & 3) * 32, col0 = (warp >> 2) * COLS;
    const uint32_t blk = smem_u32(smem) + warp * 4096u;
    constexpr int W = COLS / 4;               // 16-byte pieces of a row
    __syncwarp();
#pragma unroll
    for (int q = 0; q < W; ++q) {
        float4 o;
        unpack2(acc[2 * q], o.x, o.y);
        unpack2(acc[2 * q + 1], o.z, o.w);
        st_shared_v4(blk + lane * (W * 16) + ((q ^ (lane * W / 8 & (W - 1))) << 4), o);
    }
    __syncwarp();
#pragma unroll
    for (int k0 = 0; k0 < W; k0 += 4) {
        float4 o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = (k0 + k) * (32 / W) + lane / W, q = lane % W;
            o[k] = ld_shared_v4(blk + r * (W * 16) + ((q ^ (r * W / 8 & (W - 1))) << 4));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) p.store(c, outs[row0 + (k0 + k) * (32 / W) + lane / W], col0 + lane % W * 4, o[k]);
    }
}

// (sms: CTAs of a launch at most where kernels may not spread over all SMs, else 0)
template <int BN, bool TMA_B, class P>
inline void launch_gemm_planes(const P& p, const CUtensorMap& tmB, dim3 tiles, unsigned sms, cudaStream_t stream, int* status)
{
    allow_smem<gemm_planes_kernel<BN, P, TMA_B>>(plane_smem_bytes(BN));
    const unsigned total = tiles.x * tiles.y * tiles.z, most = sms ? sms : total;
    PlaneGrid g{0, fast_div(static_cast<int>(tiles.x)), fast_div(static_cast<int>(tiles.y))};
    for (; g.first < total; g.first += most)
        launch_after(gemm_planes_kernel<BN, P, TMA_B>, total - g.first < most ? total - g.first : most, kPlaneThreads, plane_smem_bytes(BN), stream, p, tmB, g, status);
}

// The planes of W as TMA_B copies them: dst[plane][row][pitch], row r < rows from W row src(r).  taps = 0: rows as they lie (forward; K
// columns, zeros up to the pitch); else row j * OC + oc is tap map[j] of output channel oc (deltaX: taps in the order of phases and steps).
// Words that are not the sum of their planes become NaN, which sends the tiles that read them back to W itself.
struct SplitRows { int map[64]; };
template <int>   // (defined where it is launched)
__global__ void __launch_bounds__(256) split_planes_kernel(const float* __restrict__ W, uint2* __restrict__ dst, int rows, int cols, unsigned pitch4, FastDiv by_pitch4,
                                                           FastDiv by_OC, int OC, int taps, const SplitRows map)
{
    grid_dependency_wait();
    grid_dependency_trigger();
    const unsigned total = static_cast<unsigned>(rows) * pitch4;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        unsigned r, q, from;
        by_pitch4.divmod(i, r, q);
        from = r;
        if (taps) {
            unsigned j, oc;
            by_OC.divmod(r, j, oc);
            from = oc * taps + map.map[j];
        }
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (static_cast<int>(4 * q) < cols) v = __ldg(reinterpret_cast<const float4*>(W + static_cast<size_t>(from) * cols + 4 * q));
        uint2 h, m, l;
        uint32_t lost = 0;
        split_planes(v, h, m, l, lost);
        if (lost & 0xffffu) h = make_uint2(0x7fff7fffu, 0x7fff7fffu);
        dst[i] = h; dst[static_cast<size_t>(total) + i] = m; dst[2 * static_cast<size_t>(total) + i] = l;
    }
}

// Tile and parts of the reduction of a product of `rows` x `cols` outputs over k steps, `copies` times, on this kernel (its
// launch can cut the reduction into up to `most` parts of `size` outputs each; w: elements of W where B can be split beforehand, else 0), and
// the time that takes (us): what a stage and a tile besides take in each form, as fitted to 1200 products (9 of 10 within 13 %).  The copy of
// B costs a launch and pays from a few waves on (64 x 15 x 13, 36 -> 100 channels 3x3 37 -> 34 us, 2368 x 2048 x 2304 195 -> 140).
struct PlanePlan { int bn; bool copy_b; int ksplit; double time; };
inline PlanePlan plan_planes(long long rows, int cols, long long k, long long copies, int most, double size, double w, int sms)
{
    static const struct { int bn; bool copy; double stage, wave; } forms[] = {{64, false, 0.62, 4.0}, {128, false, 0.80, 4.4}, {64, true, 0.47, 4.2}, {128, true, 0.57, 4.9}};
    const long long stages = (k + kPlaneBK - 1) / kPlaneBK;
    PlanePlan best{64, false, 1, 0};
    for (const auto& f : forms) {
        if (f.copy && !(w > 0)) continue;
        const double tiles = (double)((rows + kPlaneBM - 1) / kPlaneBM) * ((cols + f.bn - 1) / f.bn) * copies, fixed = 5.3 + (f.copy ? 1.5 + w * 10e-6 / 5 : w * 0.8e-6);
        // (of many parts, those that fill whole waves)
        auto next = [&](int ks) { return ks < 16 ? ks + 1 : (int)(((long long)(ks * tiles / sms) + 1) * sms / tiles); };
        for (int ks = 1; ks <= most && (ks == 1 || ks <= stages / 2); ks = next(ks) > ks ? next(ks) : ks + 1) {
            const double ctas = tiles * ks, waves = (double)(long long)((ctas + sms - 1) / sms);
            const double time = waves * ((stages + ks - 1) / ks * f.stage + f.wave) + fixed + (ks > 1 ? 2.1 + 0.07 * ks + (ks + 1) * size * 4e-6 / 5 : 0.0);
            if (best.time == 0 || time < best.time) best = PlanePlan{f.bn, f.copy, ks, time};
            if (ctas > 4.0 * sms) break;
        }
    }
    return best;
}

// Kernel, tile and parts for a product that is fp32 work (plane_k: steps, on average over the copies).
struct ProductPlan { GemmTile tile; int ksplit; bool copy_b; };
inline ProductPlan plan_product(long long rows, int cols, int taps, int k, long long copies, bool may_split, double size, double w, long long plane_k, int sms, int mode)
{
    const GemmTile f = pick_gemm_tile(rows, cols, copies, sms);
    const long long its = (long long)taps * ((k + kGemmBK - 1) / kGemmBK);
    const double fc = (double)((rows + f.bm - 1) / f.bm) * ((cols + f.bn - 1) / f.bn) * copies;
    // FMAs: split only where the tiles do not fill the SMs
    int fks = 1;
    if (may_split && fc < sms && its >= 8) {
        double ks = (int)(2.0 * sms / fc);
        if (ks > its / 4) ks = (double)(its / 4);
        fks = ks > 16 ? 16 : (ks < 1 ? 1 : (int)ks);
    }
    const double step = f.bn == 128 ? 3.57 : (f.bn == 32 ? 1.42 : (f.bm == 128 ? 1.93 : 1.30)), waves = fc * fks / (2.0 * sms);
    const double f_time = (waves > 1 ? waves : 1.0) * ((its + fks - 1) / fks * step + 3.1) + 6.1;
    if (mode == 0 || (mode == 1 && (long long)taps * k < 64)) return ProductPlan{f, fks, false};
    const PlanePlan p = plan_planes(rows, cols, plane_k, copies, may_split ? 16 : 1, size, w, sms);
    if (mode == 1 && f_time <= 1.05 * p.time) return ProductPlan{f, fks, false};
    return ProductPlan{GemmTile{kPlaneBM, p.bn, true}, p.ksplit, p.copy_b};
}

template <class P>
inline void launch_planes(const P& p, int bn, dim3 tiles, int sms, cudaStream_t stream, int* status, const CUtensorMap* tmB = nullptr)
{
    if constexpr (P::kCopyB) {
        if (tmB) {
            if (bn == 64) launch_gemm_planes<64, true>(p, *tmB, tiles, sms, stream, status);
            else launch_gemm_planes<128, true>(p, *tmB, tiles, sms, stream, status);
            return;
        }
    }
    if (bn == 64) launch_gemm_planes<64, false>(p, CUtensorMap{}, tiles, sms, stream, status);
    else launch_gemm_planes<128, false>(p, CUtensorMap{}, tiles, sms, stream, status);
}

}  // namespace alpha
