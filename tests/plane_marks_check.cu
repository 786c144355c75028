// Host-side check of the marks by which deltaW on bf16 planes (csrc/gemm_planes.cuh) knows columns and steps that do not exist:
// whatever the padding and the picture, neither a column nor a step past the end, nor both, may meet a pixel.
#include <cstdio>
#include "../dragon-alpha-v1.0_b200/csrc/gemm_planes.cuh"

int main()
{
    using P = alpha::PlaneDw;
    P p{};
    int bad = 0;
    const int most = (1 << 29) - 1;                    // rows of a picture: tensors have fewer than 2^31 elements, four to a pixel at least
    for (int IH : {1, 7, 1 << 20, most - 1, most})
        for (int pad : {0, 1, 2, 3, 127, 4096, 1 << 20}) {
            p.IH = IH; p.IW = 1;
            const P::BRow none{0u, P::kNone, 0};
            const P::BStep end{0u, P::kNone, 0};
            for (int y : {-pad, 0, IH - 1, IH - 1 + pad})
                bad += p.use_b(none, P::BStep{0u, y, 0}) || p.use_b(P::BRow{0u, y < 0 ? 0 : (y < 65536 ? y : 65535), 0}, end);
            bad += p.use_b(none, end);
            bad += !p.use_b(P::BRow{0u, pad, 0}, P::BStep{0u, -pad, 0}) + !p.use_b(P::BRow{0u, 0, 0}, P::BStep{0u, IH - 1, 0});
            bad += p.use_b(P::BRow{0u, 0, 0}, P::BStep{0u, -pad - 1, 0}) || p.use_b(P::BRow{0u, 1, 0}, P::BStep{0u, IH - 1, 0});
        }
    printf("%d wrong\n", bad);
    return bad != 0;
}
