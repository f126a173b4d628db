// Root-mean-square error of the short FP32 transforms (fft32.cuh) against 64 bits,
// with packed and with scalar complex sums: "radix direction packed scalar" lines.
#include "fft32.cuh"

#include <cmath>
#include <cstdio>
#include <vector>

using namespace nadia::f32;

constexpr int kSamples = 1 << 18;

// input r of sample i: uniform in (-1, 1), the same for every form
__device__ float2 value(unsigned i, unsigned r)
{
    auto mix = [](unsigned h) {
        h ^= h >> 16; h *= 0x7feb352du; h ^= h >> 15; h *= 0x846ca68bu; h ^= h >> 16;
        return h;
    };
    const unsigned a = mix(i * 64u + r), b = mix(a + 0x9e3779b9u);
    return make_float2((int)(a >> 8) * 0x1p-23f - 1.f, (int)(b >> 8) * 0x1p-23f - 1.f);
}

template <int R, bool FWD, bool PK>
__global__ void errors(double *sums)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kSamples) return;
    float2 v[R];
    for (int r = 0; r < R; ++r) v[r] = value(i, r);
    float2 u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = v[r];
    Dft<R, FWD, PK>::run(u);
    double e = 0;
    for (int k = 0; k < R; ++k) {
        double x = 0, y = 0;
        for (int r = 0; r < R; ++r) {
            double s, c;
            sincospi(2.0 * ((k * r) % R) / R, &s, &c);
            if (FWD) s = -s;
            x += v[r].x * c - v[r].y * s;
            y += v[r].x * s + v[r].y * c;
        }
        e += (u[k].x - x) * (u[k].x - x) + (u[k].y - y) * (u[k].y - y);
    }
    sums[i] = e;
}

template <int R, bool FWD, bool PK>
double rms(double *d)
{
    errors<R, FWD, PK><<<kSamples / 128, 128>>>(d);
    std::vector<double> h(kSamples);
    if (cudaMemcpy(h.data(), d, kSamples * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return -1;
    double t = 0;
    for (double e : h) t += e;
    return std::sqrt(t / kSamples / R);
}

template <int R>
void both(double *d)
{
    std::printf("%d 1 %.6e %.6e\n", R, rms<R, true, true>(d), rms<R, true, false>(d));
    std::printf("%d 0 %.6e %.6e\n", R, rms<R, false, true>(d), rms<R, false, false>(d));
}

int main()
{
    double *d = nullptr;
    if (cudaMalloc(&d, kSamples * sizeof(double)) != cudaSuccess) return 1;
    both<2>(d); both<3>(d); both<4>(d); both<5>(d); both<6>(d);
    both<8>(d); both<10>(d); both<12>(d); both<15>(d); both<16>(d);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
