// A plan's execute while operator new fails: the sum by cells chooses its shape
// with host memory, and a C caller must get a sum or an error, not an exception.
// Prints the status of the call without memory, of one with, and the largest
// difference of their displacements.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include <cuda_runtime.h>

#include "disco_b200.h"

static bool g_fail = false;

void* operator new(std::size_t n)
{
    if (g_fail) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
    const int n = 195821, chords = 24;
    const double edge = std::cbrt(n / 0.08), box[3] = { edge, edge, edge };
    std::vector<double> v[2][3];
    disco_loop loops[2] = {};
    for (int l = 0; l < 2; ++l) {
        for (int k = 0; k < chords; ++k) {
            const double t = 2.0 * 3.14159265358979323846 * k / chords;
            v[l][0].push_back(20.0 * l + 9.7 * std::cos(t));
            v[l][1].push_back(9.7 * std::sin(t));
            v[l][2].push_back(-7.0 * l);
        }
        disco_loop& d = loops[l];
        d.line = 1;
        d.n_vertices = chords;
        d.vx = v[l][0].data(); d.vy = v[l][1].data(); d.vz = v[l][2].data();
        d.cx = 20.0 * l; d.cz = -7.0 * l;
        d.phys.bx = d.phys.by = d.phys.bz = 2.5;
        d.phys.mx = 1.0; d.phys.nz = 1.0; d.phys.dS = 1.0;
    }
    std::vector<double> pos(3 * n), u[2];
    unsigned long long s = 1;
    for (double& x : pos) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        x = ((double)(s >> 11) / 9007199254740992.0 - 0.5) * edge;
    }
    double *dp = nullptr, *du = nullptr;
    if (cudaMalloc(&dp, pos.size() * 8) || cudaMalloc(&du, pos.size() * 8)) return 2;
    cudaMemcpy(dp, pos.data(), pos.size() * 8, cudaMemcpyHostToDevice);
    disco_options o;
    disco_b200_options_default(&o);
    o.images = 2;
    int status[2] = { -1, -1 };
    for (int with = 0; with < 2; ++with) {
        disco_plan* plan = nullptr;
        if (disco_b200_plan_create(loops, 2, box, &o, n, &plan)) return 3;
        cudaMemset(du, 0, pos.size() * 8);
        cudaDeviceSynchronize();
        const disco_atoms a = { dp, dp + n, dp + 2 * n, du, du + n, du + 2 * n, n };
        g_fail = with == 0;
        status[with] = disco_b200_plan_execute(plan, &a, nullptr);
        g_fail = false;
        if (disco_b200_plan_sync(plan, nullptr)) return 4;
        u[with].resize(pos.size());
        cudaMemcpy(u[with].data(), du, pos.size() * 8, cudaMemcpyDeviceToHost);
        disco_b200_plan_destroy(plan);
    }
    double diff = 0.0, most = 0.0;
    for (size_t k = 0; k < pos.size(); ++k) {
        diff = std::fmax(diff, std::fabs(u[0][k] - u[1][k]));
        most = std::fmax(most, std::fabs(u[1][k]));
    }
    std::printf("%d %d %.3e %.3e\n", status[0], status[1], diff, most);
    return 0;
}
