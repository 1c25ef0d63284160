// The FP64 primitives of the near-grazing search beside the operators that they
// stand for, on arrays from the host (test_gpu_fp64_primitives.py).
#include "../cgspline_gb300/csrc/device.cuh"

using namespace cgs;

namespace {

// a, b: operands.  got, want: 4 doubles an item.
__global__ void k_primitive(int what, uint32_t n, const double* a, const double* b, double* got, double* want)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        double *g = got + 4ull * i, *w = want + 4ull * i;
        const double x = a[i], y = b[i];
        for (int k = 0; k < 4; k++) g[k] = w[k] = 0.0;
        if (what == 0) { g[0] = quotient(x, y); w[0] = x / y; }
        if (what == 1) { g[0] = widen(float(x)); w[0] = double(float(x)); }
        if (what == 2) { g[0] = double(narrow(x)); w[0] = double(float(x)); }
        if (what == 3)
        {
            g[0] = from_ordered(ordered(x)); w[0] = x;
            g[1] = x != y && ordered(x) < ordered(y) ? 1.0 : 0.0; w[1] = x < y ? 1.0 : 0.0;
            g[2] = not_negative(x) ? 1.0 : 0.0; w[2] = x >= 0.0 ? 1.0 : 0.0;
            g[3] = not_finite(x) ? 1.0 : 0.0; w[3] = isfinite(x) ? 0.0 : 1.0;
        }
        if (what == 4)
        {
            const double2 L = make_double2(x, y), u = unit2d(L);
            // (unit2d's own length: its sum of squares contracts)
            const double l = sqrt(L.x * L.x + L.y * L.y);
            g[0] = u.x; g[1] = u.y;
            w[0] = l != 0.0 ? x / l : x; w[1] = l != 0.0 ? y / l : y;
        }
    }
}

// Nets of 16 points (32 floats each): the clip bounds of the two forms.
__global__ void k_bounds(uint32_t n, const float* nets, double* got, double* want)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        float2 p[16];
        double2 q[16];
        for (int k = 0; k < 16; k++)
        {
            p[k] = make_float2(nets[32ull * i + 2 * k], nets[32ull * i + 2 * k + 1]);
            q[k] = make_double2(p[k].x, p[k].y);
        }
        for (int side = 0; side < 2; side++)
        {
            clip_range_d([&](int k) { return make_double2(widen(p[k].x), widen(p[k].y)); }, side, got[4ull * i + 2 * side],
                         got[4ull * i + 2 * side + 1]);
            clip_range_full(q, side, want[4ull * i + 2 * side], want[4ull * i + 2 * side + 1]);
        }
    }
}

template<class F> int on_device(uint32_t n, const void* a, size_t as, const void* b, size_t bs, double* got, double* want, F&& f)
{
    uint8_t *da = nullptr, *db = nullptr;
    double* out = nullptr;
    cudaError_t e = cudaMalloc(&da, as);
    if (e == cudaSuccess) e = cudaMalloc(&db, bs);
    if (e == cudaSuccess) e = cudaMalloc(&out, 64ull * n);
    if (e == cudaSuccess) e = cudaMemcpy(da, a, as, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && b) e = cudaMemcpy(db, b, bs, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
    {
        f(da, db, out, out + 4ull * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(got, out, 32ull * n, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(want, out + 4ull * n, 32ull * n, cudaMemcpyDeviceToHost);
    cudaFree(da); cudaFree(db); cudaFree(out);
    return int(e);
}

}  // namespace

extern "C" int primitive(int what, uint32_t n, const double* a, const double* b, double* got, double* want)
{
    return on_device(n, a, 8ull * n, b, 8ull * n, got, want, [&](uint8_t* da, uint8_t* db, double* g, double* w) {
        k_primitive<<<512, 128>>>(what, n, reinterpret_cast<double*>(da), reinterpret_cast<double*>(db), g, w);
    });
}

extern "C" int bounds(uint32_t n, const float* nets, double* got, double* want)
{
    return on_device(n, nets, 128ull * n, nullptr, 16, got, want, [&](uint8_t* da, uint8_t*, double* g, double* w) {
        k_bounds<<<512, 64>>>(n, reinterpret_cast<float*>(da), g, w);
    });
}
