// A program that resets the device between uses of the library; a handle of the first
// context is left alive across the reset, the others are destroyed before it.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "hmg.h"

static void check(hmg_status st, const char* what)
{
    if (st != HMG_OK) {
        fprintf(stderr, "%s: %s\n", what, hmg_last_error());
        exit(1);
    }
}

static hmg_matrix* build(const std::vector<double>& p, int n)
{
    hmg_matrix* h = nullptr;
    check(hmg_create(&h, n, n, 2, 0, nullptr), "hmg_create");
    for (int set = 0; set < 2; set++) check(hmg_set_points(h, set, p.data(), 0), "hmg_set_points");
    check(hmg_setup(h, 1.5, 64, 50, 0, 0, 1), "hmg_setup");
    check(hmg_set_kernel(h, HMG_KERNEL_GAUSSIAN, 0.05, 0.0), "hmg_set_kernel");
    check(hmg_precompute_aca(h, 64, 1e-8, HMG_PREC_FP64), "hmg_precompute_aca");
    check(hmg_precompute_dense(h, HMG_PREC_FP64), "hmg_precompute_dense");
    return h;
}

int main()
{
    const int n = 5000;
    std::vector<double> p(2 * n), x(n), y[3];
    unsigned s = 1;
    auto rnd = [&]() { return (s = s * 1664525u + 1013904223u) / 4294967296.0; };
    for (double& v : p) v = rnd();
    for (double& v : x) v = 2.0 * rnd() - 1.0;
    hmg_matrix* left = nullptr;
    for (int i = 0; i < 3; i++) {
        y[i].resize(n);
        hmg_matrix* h = build(p, n);
        check(hmg_matvec_host(h, x.data(), y[i].data()), "hmg_matvec_host");
        if (i == 0) left = h;  // its memory ends with the context
        else check(hmg_destroy(h), "hmg_destroy");
        if (i < 2 && cudaDeviceReset() != cudaSuccess) return 2;
    }
    (void)left;
    for (int i = 0; i < n; i++)
        if (y[0][i] != y[1][i] || y[0][i] != y[2][i]) return 3;
    printf("equal\n");
    return 0;
}
