// The closure's calls across a device reset: the blocks that a program
// allocates after it keep what the program wrote there, whatever the library
// held before it.
//   mlp_reset_check  -> exit 1 on a difference
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "des_gpu.h"

static const long long n = 300;
static std::vector<float> x(n * DES_MLP_IN), t(n * DES_MLP_OUT, 0.5f);
static des_mlp net;

static int call(std::vector<float> &y)
{
    des_mlp g;
    double loss = 0;
    y.assign(n * DES_MLP_OUT, 0.f);
    return des_mlp_forward(&net, x.data(), n, y.data()) || des_mlp_loss_grad(&net, x.data(), t.data(), n, &loss, &g);
}

struct Blocks {
    std::vector<unsigned char *> p;
    std::vector<size_t> size;
    bool fill()
    {
        for (int k = 0; k < 96; ++k) {
            unsigned char *q = nullptr;
            const size_t b = k % 3 ? 46160 : 3 << 20;
            if (cudaMalloc(&q, b) || cudaMemset(q, 0xa5, b)) return false;
            p.push_back(q);
            size.push_back(b);
        }
        return cudaDeviceSynchronize() == cudaSuccess;
    }
    bool intact()
    {
        for (size_t k = 0; k < p.size(); ++k) {
            std::vector<unsigned char> h(size[k]);
            if (cudaMemcpy(h.data(), p[k], size[k], cudaMemcpyDeviceToHost)) return false;
            for (unsigned char c : h)
                if (c != 0xa5) return false;
        }
        return true;
    }
};

int main()
{
    std::memset(&net, 0, sizeof net);
    unsigned s = 1;
    auto draw = [&] { return (float)((s = s * 1664525u + 1013904223u) >> 8) / 16777216.f - 0.5f; };
    for (float *w = &net.w1[0][0]; w < &net.in_mean[0]; ++w) *w = draw();
    for (float &v : x) v = draw();
    std::vector<float> first, again;
    if (call(first)) return printf("first call failed\n"), 1;
    // a thread that called before the reset and ends after it
    if (cudaDeviceReset()) return printf("reset failed\n"), 1;
    {
        Blocks b;
        if (!b.fill()) return printf("allocation failed\n"), 1;
        if (call(again) || again != first) return printf("the call after the reset differs\n"), 1;
        if (!b.intact()) return printf("a block of the program's was overwritten\n"), 1;
    }
    int rc = 0;
    Blocks b;
    std::thread([&] {
        std::vector<float> y;
        rc = call(y) || cudaDeviceReset() || !b.fill();
    }).join();
    if (rc || !b.intact()) return printf("a thread's end took a block of the program's\n"), 1;
    for (unsigned char *p : b.p)
        if (cudaFree(p)) return printf("a block of the program's was gone\n"), 1;
    printf("ok\n");
    return 0;
}
