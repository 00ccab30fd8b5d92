// What the convolution launchers must refuse before they launch anything; needs no GPU.
// Prints one line a failure, exits 0 when there is none.
#include "../../isaac_b200/csrc/isaacb_conv.h"

#include <cstdio>
#include <vector>

using namespace isaacb;

int main()
{
    std::setvbuf(stdout, nullptr, _IONBF, 0);
    int bad = 0;
    auto refused = [&](bool launched, const char* what) {
        if(launched)
        {
            std::printf("not refused: %s\n", what);
            ++bad;
        }
    };
    // a concatenation that the row-tile kernel has no room for, while the general kernel,
    // which knows no second input, has
    ConvGemmParams p{};
    p.B = 1;
    p.H = p.Ho = 4;
    p.W = p.Wo = 200;
    p.Cg = 320;
    p.Cout = p.Npad = 256;
    p.Kpad = 320;
    p.ks = p.stride = 1;
    alignas(16) static unsigned char memory[64];
    p.x = p.w = p.xUp = reinterpret_cast<const __nv_bfloat16*>(memory);
    p.y = reinterpret_cast<__nv_bfloat16*>(memory);
    p.upC = 160;
    p.upInH = 2;
    p.upInW = 100;
    if(!row_tiles_apply(p) || conv_gemm_smem(p.Npad, p.Kpad) > 227 * 1024)
    {
        std::printf("the sizes no longer separate the two kernels\n");
        return 1;
    }
    refused(launch_conv_gemm(p, nullptr), "a concatenation without room for the row-tile kernel");
    // a concatenation of a shape that the row-tile kernel does not take at all
    p.Cg = p.Kpad = 64;
    p.Npad = p.Cout = 32;
    p.upC = 20;
    refused(launch_conv_gemm(p, nullptr), "a concatenation that is not in 8-channel groups");
    // more layers than the table holds, and none
    std::vector<WgradParams> layers(kWgradLayers + 1);
    for(auto& l : layers)
    {
        l.B = l.H = l.W = l.Ho = l.Wo = l.ks = l.stride = 1;
        l.Cin = l.Cout = l.Npad = l.Mtot = 16;
    }
    refused(launch_conv_wgrad(layers.data(), kWgradLayers + 1, nullptr), "more layers than kWgradLayers");
    refused(launch_conv_wgrad(layers.data(), 0, nullptr), "no layer");
    return bad ? 1 : 0;
}
