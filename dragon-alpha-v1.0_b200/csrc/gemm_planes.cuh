// The products of gemm_f32.cuh on the tensor cores, at fp32 accuracy.
//
// An fp32 word is the exact sum of three bf16 words, x = h + m + l (the upper 16 bits, the upper 16 bits of what is left, the rest: 8
// bits of significand each), and of the nine products of two such sums the six that matter are formed by tcgen05.mma kind::f16:
// hh in one accumulator; hm, mh, mm, hl, lh, all below 2^-7 of it, in another.  What is dropped (ml, lm, ll) is below 2^-23 of a product.
// The tensor core truncates as it adds to an accumulator, about 2^-24 of it an instruction, which over a long sum would cost more
// than fp32 FMAs do: after every 64 reduction steps (four instructions into the hh accumulator) the partial sum is added to running
// sums in registers, rounded to nearest, and the accumulator starts anew.  The errors are given at plan_product.
//
// Bound: 388 clocks of MMAs per 16 steps of a 128 x 128 tile, as much as the 3xTF32 kernels issue per step, against which shared
// memory takes 96 KB of plane stores and operand reads per 32 steps (40 KB a step in MMAs of 256, 256, 128 and 128 columns; six of 128 would
// read 48).  2048 x 2048 x 2052: 127 TFLOP/s, some 1900 clocks for the 776 of MMAs a stage; the issuing thread's share of the issue slots and
// the stores of 16 warps in the MMAs' way are what is left (measured with clocks around every MMA).
//
// A CTA of 544 threads forms 128 x BN outputs of a policy P (see gemm_f32.cuh; a stage is 32 steps of it):
//   warps 0-15  in two groups that take alternate stages, so that the loads of one are in flight while the other splits: load the words of
//               a stage, split them and store the planes of both operands in shared memory as the MMA reads them - rows of 32 steps where
//               the operand's memory runs along k (K-major), rows of 32 columns where it does not (MN-major; no transposition) - with the
//               64-byte swizzle; a warp's four rows of eight words are 256 consecutive bytes of a plane: no bank conflicts.  They also add
//               up the flushed sums, a quarter of the columns each, and store the result.  96 registers a thread allow no more: with more
//               live words or sums they spill, and what spills goes to L2 (shared memory leaves no L1; 44 TFLOP/s).
//   warp 16     issues the MMAs.  The three planes of B are neighbouring rows (or column blocks) of one operand, so that h x [m l], m x [h m]
//               are one MMA each, and with BN = 64 also h x [h m l].
// hh accumulates in two column blocks in turn, so that one is read while the other fills.
// Where a sum comes out as Inf or NaN (operands that are, or that overflow a plane) or so small that a plane's last bits may have
// been lost to underflow, the tile is formed once more by FMAs, as gemm_f32_kernel forms it.
#pragma once
#include "gemm_f32.cuh"
#include "sm100_ptx.cuh"

namespace alpha {

constexpr int kPlaneThreads = 544, kPlaneBM = 128, kPlaneBK = 32, kPlaneRing = 4;

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

// x = h + m + l: the planes of four consecutive elements, eight bytes each.
__device__ __forceinline__ void split_planes(const float4& v, uint2& h, uint2& m, uint2& l)
{
    auto hi2 = [](float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); };
    auto cut = [](float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); };
    float r0, r1, r2, r3, t0, t1, t2, t3;
    unpack2(sub2(pack2(v.x, v.y), pack2(cut(v.x), cut(v.y))), r0, r1);
    unpack2(sub2(pack2(v.z, v.w), pack2(cut(v.z), cut(v.w))), r2, r3);
    unpack2(sub2(pack2(r0, r1), pack2(cut(r0), cut(r1))), t0, t1);
    unpack2(sub2(pack2(r2, r3), pack2(cut(r2), cut(r3))), t2, t3);
    h = make_uint2(hi2(v.x, v.y), hi2(v.z, v.w));
    m = make_uint2(hi2(r0, r1), hi2(r2, r3));
    l = make_uint2(hi2(t0, t1), hi2(t2, t3));
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

// The whole tile by FMAs, in column slices of 64.
template <int BN, class P>
__device__ __noinline__ void gemm_planes_again(const P& p, void* shared)
{
    typename P::Cta c;
    p.cta(c, kPlaneBM, BN);
    for (int x = 0; x < BN; x += 64) {
        typename P::Cta part = c;
        part.n0 += x;
        gemm_f32_tile<kPlaneBM, 64, 8, 4>(p, part, *static_cast<GemmShared<kPlaneBM, 64, P>*>(shared));
    }
}

template <int BN, class P>
__global__ void __launch_bounds__(kPlaneThreads, 1) gemm_planes_kernel(const __grid_constant__ P p, int* status)
{
    static_assert(BN == 64 || BN == 128, "tile shape");
    constexpr int NA = kPlaneBM / 32, NB = BN / 32, COLS = BN / 4;      // words of a thread in a stage; columns of a warp
    constexpr uint32_t kPlaneA = kPlaneBM * kPlaneBK * 2, kPlaneB = BN * kPlaneBK * 2, kStage = plane_stage_bytes(BN), kTmem = BN == 64 ? 256 : 512;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bars[2 * kPlaneRing + 2];
    __shared__ uint32_t tmem_holder;
    __shared__ typename P::Cta c;                            // (in registers or local memory it would cost the loops)
    __shared__ int work;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full_a = smem_u32(bars), done_a = full_a + 8 * kPlaneRing, free_a = done_a + 8 * kPlaneRing;
    if (tid == 0) {
        for (int i = 0; i < kPlaneRing; ++i) {
            mbar_init(&bars[i], 8);                      // a stage is staged: one arrival per warp of its group
            mbar_init(&bars[kPlaneRing + i], 1);         // its MMAs are done
        }
        mbar_init(&bars[2 * kPlaneRing], 16);            // an hh accumulator has been read by all warps
        mbar_init(&bars[2 * kPlaneRing + 1], 16);
        fence_barrier_init();
        typename P::Cta mine;
        work = p.cta(mine, kPlaneBM, BN);
        c = mine;
    }
    if (warp == 16) {
        tmem_alloc(&tmem_holder, kTmem);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    grid_dependency_wait();
    __syncthreads();
    grid_dependency_trigger();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_holder;

    const int stages = work && c.it1 > c.it0 ? (c.it1 - c.it0 + 1) >> 1 : 0;
    bool ok = true, again = false;
    unsigned long long acc[COLS / 2];
#pragma unroll
    for (int x = 0; x < COLS / 2; ++x) acc[x] = 0ull;
    // tensor memory: [hh of even windows][hm + mh][hl + mm + lh][hh of odd windows]
    constexpr uint32_t kSide = BN, kOdd = 3 * BN;

    if (warp >= 16) {
        if (warp == 16 && lane == 0 && stages) {
            constexpr uint32_t dhi = (512u >> 4) | (1u << 14) | (static_cast<uint32_t>(kSwizzle64B) << 29);
            constexpr uint32_t a_k = P::kAk ? 2u : 64u, b_k = P::kBk ? 2u : 64u;      // 16 steps further, in 16-byte units
            constexpr uint32_t i1 = make_idesc_bf16(128, BN, !P::kAk, !P::kBk), i2 = make_idesc_bf16(128, 2 * BN, !P::kAk, !P::kBk),
                               i3 = make_idesc_bf16(128, BN == 64 ? 192 : 128, !P::kAk, !P::kBk);
            constexpr uint32_t pa = kPlaneA >> 4, pb = kPlaneB >> 4;
            const uint32_t a_lo0 = smem_desc_lo(smem_u32(smem), P::kAk ? 16u : 2048u), b_lo0 = smem_desc_lo(smem_u32(smem) + 3 * kPlaneA, P::kBk ? 16u : 2048u);
            const uint32_t side = tmem_base + kSide;
            typename P::Cursor cur = p.plane_begin(c);
            auto full = [&](int s) { return full_a + 8 * (s % kPlaneRing); };
            auto freed = [&](int s) { return free_a + 8 * (s >> 1 & 1); };    // (asked at the first stage of a window)
            bool staged = false, read = false;       // stage s is known to be staged, the accumulator of its window to be read
            for (int s = 0; s < stages; ++s) {
                const uint32_t slot = s % kPlaneRing, window = s >> 1, d = tmem_base + (window & 1 ? kOdd : 0u);
                if (!staged) ok = mbar_wait_a(full(s), (s / kPlaneRing) & 1);
                if (ok && !read && !(s & 1) && window >= 2) ok = mbar_wait_a(freed(s), ((window >> 1) - 1) & 1);
                if (!ok) { report(status, kStatusMmaTimeout); break; }
                tc_fence_after_sync();
                const bool two = p.plane_left(cur) > 16;
                const uint32_t a = a_lo0 + slot * (kStage >> 4), b = b_lo0 + slot * (kStage >> 4);
                const uint32_t keep = s & 1, keep_side = s ? 1u : 0u;
                // what the next stage waits for, asked while the queue still holds MMAs of this one
                auto look_ahead = [&]() {
                    p.plane_next(c, cur);
                    const int n = s + 1;
                    staged = mbar_test_a(full(n), (n / kPlaneRing) & 1);
                    read = !(n & 1) && n >= 4 && mbar_test_a(freed(n), ((n >> 2) - 1) & 1);
                };
                // straight-line code: address arithmetic between two MMAs would cost the issuing thread as much as an MMA takes
                if constexpr (BN == 64) {
                    // small products: [hm + mh][hl + mm + lh]
                    auto step = [&](auto merged_, auto k_, uint32_t keep, uint32_t keep_side) {
                        constexpr uint32_t ka = decltype(k_)::value * a_k, kb = decltype(k_)::value * b_k;
                        if constexpr (decltype(merged_)::value) {
                            mma_bf16_ss2_imm<ka, kb>(d, a, dhi, b, dhi, i3, 1u);
                        } else {
                            mma_bf16_ss2_imm<ka, kb>(d, a, dhi, b, dhi, i1, keep);
                            mma_bf16_ss2_imm<ka, kb + pb>(side, a, dhi, b, dhi, i2, keep_side);
                        }
                        mma_bf16_ss2_imm<ka + pa, kb>(side, a, dhi, b, dhi, i2, 1u);
                        mma_bf16_ss2_imm<ka + 2 * pa, kb>(side + 64, a, dhi, b, dhi, i1, 1u);
                    };
                    using First = std::integral_constant<uint32_t, 0>; using Second = std::integral_constant<uint32_t, 1>;
                    if (window & 1) {
                        step(std::false_type{}, First{}, keep, 1u);
                        look_ahead();
                        if (two) step(std::false_type{}, Second{}, 1u, 1u);
                    } else if (keep) {
                        step(std::true_type{}, First{}, 1u, 1u);
                        look_ahead();
                        if (two) step(std::true_type{}, Second{}, 1u, 1u);
                    } else {
                        step(std::false_type{}, First{}, 0u, keep_side);
                        look_ahead();
                        if (two) step(std::true_type{}, Second{}, 1u, 1u);
                    }
                } else {
                    auto step = [&](auto k_, uint32_t keep, uint32_t keep_side) {
                        constexpr uint32_t ka = decltype(k_)::value * a_k, kb = decltype(k_)::value * b_k;
                        // small products: [hm + mh][hl + mm + lh]
                        mma_bf16_ss2_imm<ka, kb + pb>(side, a, dhi, b, dhi, i2, keep_side);
                        mma_bf16_ss2_imm<ka + pa, kb>(side, a, dhi, b, dhi, i2, 1u);
                        mma_bf16_ss2_imm<ka + 2 * pa, kb>(side + BN, a, dhi, b, dhi, i1, 1u);
                        mma_bf16_ss2_imm<ka, kb>(d, a, dhi, b, dhi, i1, keep);
                    };
                    step(std::integral_constant<uint32_t, 0>{}, keep, keep_side);
                    look_ahead();
                    if (two) step(std::integral_constant<uint32_t, 1>{}, 1u, 1u);
                }
                mma_commit_a(done_a + 8 * slot);
            }
        }
        __syncwarp();
    } else {
        if (stages) {
        const int group = warp >> 3, t = tid & 255;          // two groups of 256 threads take alternate stages
        typename P::PlaneRow ra[NA];
        if (P::kAk)
#pragma unroll
            for (int i = 0; i < NA; ++i) ra[i] = p.plane_row(c, plane_col<kPlaneBM, P::kAk>(t, i));
        const uint32_t off_a = smem_u32(smem) + plane_offset<kPlaneBM, P::kAk>(t), off_b = smem_u32(smem) + 3 * kPlaneA + plane_offset<BN, P::kBk>(t);
        const float* base_a = p.plane_a_base(c, plane_col<kPlaneBM, P::kAk>(t, 0), plane_k<kPlaneBM, P::kAk>(t, 0));
        const float* base_b = p.plane_b_base(c, plane_col<BN, P::kBk>(t, 0), plane_k<BN, P::kBk>(t, 0));
        uint32_t in = 0;                                     // words whose row or column exists
#pragma unroll
        for (int i = 0; i < NA; ++i) in |= (p.plane_a_in(c, plane_col<kPlaneBM, P::kAk>(t, i)) ? 1u : 0u) << i;
#pragma unroll
        for (int i = 0; i < NB; ++i) in |= (p.plane_b_in(c, plane_col<BN, P::kBk>(t, i)) ? 1u : 0u) << (8 + i);
        typename P::Cursor cur = p.plane_begin(c);
        float4 va[NA], vb[NB];
        auto load = [&]() {
#pragma unroll
            for (int i = 0; i < NA; ++i)
                va[i] = p.plane_a(cur, base_a, ra[i], i, in >> i & 1u, plane_k<kPlaneBM, P::kAk>(t, i), plane_dk<kPlaneBM>());
#pragma unroll
            for (int i = 0; i < NB; ++i) vb[i] = p.plane_b(cur, base_b, i, in >> (8 + i) & 1u, plane_k<BN, P::kBk>(t, i), plane_dk<BN>());
        };
        const uint32_t lanes = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (warp >> 2) * COLS;
        // acc += the warp's columns of a column block
        auto add_columns = [&](uint32_t from) {
#pragma unroll
            for (int x = 0; x < COLS; x += 16) {
                uint32_t v[16];
                tmem_ld_32x16(lanes + from + x, v);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 16; q += 2) acc[(x + q) / 2] = add2(acc[(x + q) / 2], pack2(__uint_as_float(v[q]), __uint_as_float(v[q + 1])));
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
        if (group) p.plane_next(c, cur);
        if (group < stages) load();
        for (int s = group; s < stages; s += 2) {
            // two windows back: its MMAs are done, or nearly
            if (s >= 4 && !flush(flushed++)) break;
            if (s >= kPlaneRing && !wait_done(s - kPlaneRing)) break;
            const uint32_t at_a = off_a + (s % kPlaneRing) * kStage, at_b = off_b + (s % kPlaneRing) * kStage;
            if (P::kTail) {
                const int steps = p.plane_left(cur);
                if (steps < 32) {
                    if (P::kAk)
#pragma unroll
                        for (int i = 0; i < NA; ++i) keep_first(va[i], steps - plane_k<kPlaneBM, true>(t, i));
                    if (P::kBk)
#pragma unroll
                        for (int i = 0; i < NB; ++i) keep_first(vb[i], steps - plane_k<BN, true>(t, i));
                }
            }
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                uint2 h, m, l;
                split_planes(va[i], h, m, l);
                const uint32_t at = at_a + i * plane_step<kPlaneBM, P::kAk>();
                st_shared_v2(at, h); st_shared_v2(at + kPlaneA, m); st_shared_v2(at + 2 * kPlaneA, l);
            }
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                uint2 h, m, l;
                split_planes(vb[i], h, m, l);
                const uint32_t at = at_b + i * plane_step<BN, P::kBk>();
                st_shared_v2(at, h); st_shared_v2(at + kPlaneB, m); st_shared_v2(at + 2 * kPlaneB, l);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_a(full_a + 8 * (s % kPlaneRing));
            // (not before the fence, which waits for loads in flight)
            if (s + 2 < stages) {
                p.plane_next(c, cur);
                p.plane_next(c, cur);
                load();
            }
        }
        const int windows = (stages + 1) >> 1;
        while (ok && flushed < windows) flush(flushed++);
        if (ok) {
            tc_fence_after_sync();
            add_columns(kSide);
            add_columns(kSide + BN);
            // what may not have survived the split
#pragma unroll
            for (int x = 0; x < COLS / 2; ++x) {
                float a, b;
                unpack2(acc[x], a, b);
                a = fabsf(a); b = fabsf(b);
                again = again || !(a <= 3.402823466e38f) || !(b <= 3.402823466e38f) || (a < 1e-28f && a > 0.f) || (b < 1e-28f && b > 0.f);
            }
        }
        }
        tc_fence_before_sync();
    }
    again = __syncthreads_or(again) != 0;     // every MMA has completed: shared memory is free
    if (warp == 16) tmem_dealloc(tmem_base, kTmem);
    if (!work || warp >= 16) return;
    if (again) {
        if (warp < 8) gemm_planes_again<BN>(p, smem);
        return;
    }
    if (!ok) return;
    // A lane holds a row; written from the registers, an instruction would touch 32 rows for 16 bytes each.  The warp's block of 32
    // columns goes through 4 KB of shared memory and leaves as whole 128-byte pieces, four rows per instruction.
    const int row0 = (warp & 3) * 32, col0 = (warp >> 2) * COLS;
    const unsigned long long own = reinterpret_cast<unsigned long long>(p.row_c(c, row0 + lane).p);
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
    for (int k = 0; k < W; ++k) {
        const int r = k * (32 / W) + lane / W, q = lane % W;
        const float4 o = ld_shared_v4(blk + r * (W * 16) + ((q ^ (r * W / 8 & (W - 1))) << 4));
        typename P::RowC rc;
        rc.p = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, own, r));
        p.store(c, rc, col0 + q * 4, o);
    }
}

template <int BN, class P>
inline void launch_gemm_planes(const P& p, dim3 grid, cudaStream_t stream, int* status)
{
    static bool attr_done = false;   // per instantiation; the attribute is per function, any device
    if (!attr_done) {
        cudaFuncSetAttribute(gemm_planes_kernel<BN, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, plane_smem_bytes(BN));
        attr_done = true;
    }
    launch_after(gemm_planes_kernel<BN, P>, grid, kPlaneThreads, plane_smem_bytes(BN), stream, p, status);
}

// Tile, kernel and parts of the reduction for a product of `rows` x `cols` outputs over `taps` x `k` steps, `copies` times (may_split: its
// launch can cut the reduction into up to 16 parts; `size` outputs in all).  Both kernels are predicted from what was measured (us; 56
// products of 1e5 to 1e10 FMAs, deltaX layers, FullConnect, batches, each within 12 % of its prediction, the choice on average 1.01 times
// as long as the better one):
//   planes  per wave of one CTA an SM 5.9 and for every stage 0.64 (64 columns) or 1.06 (128)
//   FMAs    per wave of two CTAs an SM 3.1 and for every 16 steps what its tile takes (3.6 us for 128 x 128: 42 TFLOP/s)
// 2048 x 2048 x 2052: 471 -> 136 us (127 TFLOP/s); 36848 x 384 x 604: 391 -> 174; 22275 x 248 over 9 x 84: 278 -> 107; 55404 x 272
// over 9 x 4 (whole stages a tap) 164 and 137 us; 49600 x 8 over 4 x 4, four phases: 49 and 100 us.
// Error, 2-norm against 64 bits (normal inputs): 50 steps 0.9e-7 on both, 252: 2.0e-7 -> 1.1e-7, 900: 5.3e-7 -> 1.4e-7, 2052: 1.6e-7; 20 steps
// 0.6e-7 and 0.8e-7, so that shorter sums than 64 steps stay with the FMAs.
struct ProductPlan { GemmTile tile; int ksplit; };
inline ProductPlan plan_product(long long rows, int cols, int taps, int k, long long copies, bool may_split, double size, int sms, int mode)
{
    const GemmTile f = pick_gemm_tile(rows, cols, copies, sms);
    const long long its = (long long)taps * ((k + kGemmBK - 1) / kGemmBK), stages = (long long)taps * ((k + kPlaneBK - 1) / kPlaneBK);
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
    if (mode == 0 || (mode == 1 && (long long)taps * k < 64)) return ProductPlan{f, fks};
    const GemmTile t{kPlaneBM, cols <= 64 ? 64 : 128, true};
    const double pc = (double)((rows + t.bm - 1) / t.bm) * ((cols + t.bn - 1) / t.bn) * copies;
    int pks = 1;
    double p_time = 0;
    for (int ks = 1; ks <= 16 && (ks == 1 || (may_split && ks <= stages / 2)); ++ks) {
        const double w = pc * ks, full = (long long)((w + sms - 1) / sms);
        const double time = full * ((stages + ks - 1) / ks * (t.bn == 64 ? 0.64 : 1.06) + 5.9) + 6.6 + (ks > 1 ? 2.8 + (ks + 1) * size * 4e-6 / 5 : 0.0);
        if (ks == 1 || time < p_time) { p_time = time; pks = ks; }
    }
    if (mode == 1 && f_time <= p_time) return ProductPlan{f, fks};
    return ProductPlan{t, pks};
}

template <class P>
inline void launch_product(const P& p, const GemmTile& t, dim3 grid, cudaStream_t stream, int* status)
{
    if (!t.planes) launch_gemm_f32(p, t, grid, stream);
    else if (t.bn == 64) launch_gemm_planes<64>(p, grid, stream, status);
    else launch_gemm_planes<128>(p, grid, stream, status);
}

}  // namespace alpha
