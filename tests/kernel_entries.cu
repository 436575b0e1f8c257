// Host entries to single launchers of libtracer_gpu.so, for the tests: host arrays in and
// out, one launch sequence each.  Built by tests/kernel_entries.py against the library.
#include "tc_device.cuh"
#include "tc_nn.h"

#include <vector>

namespace {
struct Buf {
    std::vector<void*> p;
    ~Buf() {
        for (void* q : p) cudaFree(q);
    }
    template <class T>
    T* put(const T* host, size_t n) {
        void* d = nullptr;
        if (cudaMalloc(&d, n * sizeof(T)) != cudaSuccess) return nullptr;
        p.push_back(d);
        if (host) cudaMemcpy(d, host, n * sizeof(T), cudaMemcpyHostToDevice);
        else cudaMemset(d, 0, n * sizeof(T));
        return (T*)d;
    }
};
Lay layout(int a, int b) {
    Lay L;
    L.a = a;
    L.b = b;
    L.ld = (a + 1 + 2 * SP + 31) / 32 * 32;
    L.nk = b + 1 + 2 * SP;
    L.plane = (size_t)L.ld * L.nk;
    return L;
}
}  // namespace

extern "C" {

// AB: (2 kl + ku + 1) x n, factored in place; info[0]: first zero pivot, info[1]: a wait gave up
int entry_lu(double* AB, int n, int kl, int ku, int* ipiv, int* info, int no_cluster) {
    Buf m;
    const size_t len = (size_t)(2 * kl + ku + 1) * n;
    double* d = m.put(AB, len);
    int* pv = m.put((const int*)nullptr, (size_t)n);
    DevScalars* ds = m.put((const DevScalars*)nullptr, 1);
    if (!d || !pv || !ds) return 2;
    Level lv{};
    lv.no_cluster = no_cluster;
    launch_coarse_lu(0, lv, d, pv, n, kl, ku, ds);
    DevScalars hs;
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    cudaMemcpy(AB, d, len * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(ipiv, pv, n * sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(&hs, ds, sizeof(hs), cudaMemcpyDeviceToHost);
    info[0] = hs.lu_info;
    info[1] = hs.visit_timeout;
    return 0;
}

int entry_inverse(const double* AB, const int* ipiv, int n, int kl, int ku, double* inv) {
    Buf m;
    const double* d = m.put(AB, (size_t)(2 * kl + ku + 1) * n);
    const int* pv = m.put(ipiv, (size_t)n);
    double* out = m.put((const double*)nullptr, (size_t)n * n);
    if (!d || !pv || !out) return 2;
    launch_coarse_inverse(0, d, pv, n, kl, ku, out);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    cudaMemcpy(inv, out, sizeof(double) * n * n, cudaMemcpyDeviceToHost);
    return 0;
}

// rhs, x: n = (a + 1)(b + 1) values, q = (b + 1) i + k; only the interior's are read and written
int entry_solve(const double* AB, const int* ipiv, const double* rowb, int a, int b, int kl, int ku,
                const double* rhs, double* x, int fp32, int no_cluster, int* timeout) {
    Buf m;
    const int n = (a + 1) * (b + 1);
    Level lv{};
    lv.L = layout(a, b);
    lv.no_cluster = no_cluster;
    const double* d = m.put(AB, (size_t)(2 * kl + ku + 1) * n);
    const int* pv = m.put(ipiv, (size_t)n);
    const double* rb = m.put(rowb, (size_t)n);
    int* to = m.put((const int*)nullptr, 1);
    std::vector<double> r(lv.L.plane, 0.0);
    std::vector<float> rf(lv.L.plane, 0.f);
    for (int i = 1; i < a; i++)
        for (int k = 1; k < b; k++) {
            r[IX(lv.L, i, k)] = rhs[(b + 1) * i + k];
            rf[IX(lv.L, i, k)] = (float)rhs[(b + 1) * i + k];
        }
    lv.rhs = m.put(r.data(), r.size());
    lv.rhs32 = m.put(rf.data(), rf.size());
    double* e = m.put((const double*)nullptr, lv.L.plane);
    float* e32 = m.put((const float*)nullptr, lv.L.plane);
    if (!d || !pv || !rb || !to || !lv.rhs || !lv.rhs32 || !e || !e32) return 2;
    if (fp32) launch_coarse_solve32(0, lv, d, pv, rb, n, kl, ku, e32, 0, to);
    else launch_coarse_solve(0, lv, d, pv, rb, n, kl, ku, e, 0, to);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    cudaMemcpy(timeout, to, sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(r.data(), e, r.size() * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(rf.data(), e32, rf.size() * sizeof(float), cudaMemcpyDeviceToHost);
    for (int i = 1; i < a; i++)
        for (int k = 1; k < b; k++)
            x[(b + 1) * i + k] = fp32 ? (double)rf[IX(lv.L, i, k)] : r[IX(lv.L, i, k)];
    return 0;
}

// whether a level of a x b cells takes the one-launch viscosity filter
int entry_vis_filter_fits(int a, int b, int stretched, int interpolate) {
    Level lv{};
    lv.L = layout(a, b);
    lv.c.M.on = stretched;
    return vis_filter_fits(lv, interpolate) ? 1 : 0;
}

// whether a visit of a x b cells with the per-point factor takes the row-strip kernel
int entry_visit_cluster_beats_tiles(int a, int b, int nsweeps) {
    return visit_cluster_beats_tiles(layout(a, b), nsweeps) ? 1 : 0;
}

// x [nb][H][W][x_tot], dz [nb][H][W][cout] BF16; part: entry_wgrad_splits x cout x 9 x cin
int entry_wgrad_splits(int nb, int H, int W, int cin) { return wgrad_splits(nb, H, W, cin); }
int entry_wgrad(const uint16_t* x, int x_tot, int x_off, int cin, const uint16_t* dz, int cout, int nb, int H, int W,
                float* part) {
    Buf m;
    const size_t np = (size_t)nb * H * W, len = (size_t)wgrad_splits(nb, H, W, cin) * cout * 9 * cin;
    const uint16_t* dx = m.put(x, np * x_tot);
    const uint16_t* dd = m.put(dz, np * cout);
    float* out = m.put((const float*)nullptr, len);
    int* fail = m.put((const int*)nullptr, 1);
    if (!dx || !dd || !out || !fail) return 2;
    const int r = wgrad_launch(0, (const __nv_bfloat16*)dx, x_tot, x_off, cin, (const __nv_bfloat16*)dd, cout, nb, H, W,
                               out, fail);
    if (r != 0) return 10 + r;
    int f = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    cudaMemcpy(&f, fail, sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(part, out, len * sizeof(float), cudaMemcpyDeviceToHost);
    return f ? 3 : 0;
}
}
