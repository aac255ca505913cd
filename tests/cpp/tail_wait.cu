// The coarse end of the V-cycle (k_tail.cu) where its tables never arrive: the
// barrier of the first copies is told of 16 bytes more than come, so that the wait
// runs out, and the tables hold offsets far outside shared memory, as memory that
// no copy has written may. The kernel has to come back with the error recorded and
// the first level's x untouched; with the right counts and tables it then solves.
// Prints one line a launch: ctas, err, breakdown, done, x changed.
#include <cstdio>
#include <cstring>
#include <vector>

#include "kernels.h"

using namespace ct;

namespace {
struct Stack {
    std::vector<LevelView<float>> v;
    std::vector<float*> owned;
    float* array(const Geo& g, float value) {
        const size_t n = (size_t)g.plane * g.nz;
        std::vector<float> h(n, 0.0f);
        for (int l = 0; l < g.nz; ++l)
            for (int j = 0; j < g.ny; ++j)
                for (int i = 0; i < g.nx; ++i) h[(size_t)l * g.plane + scol(g, i, j)] = value;
        float* d = nullptr;
        if (cudaMalloc(&d, n * 4) != cudaSuccess) return nullptr;
        cudaMemcpy(d, h.data(), n * 4, cudaMemcpyHostToDevice);
        owned.push_back(d);
        return d;
    }
    Stack(int nx, int ny, int nz) {
        for (;;) {
            LevelView<float> L;
            std::memset(&L, 0, sizeof L);
            L.g = geo_of(nx, ny, nz);
            L.gE = array(L.g, 0.0f);
            L.gN = array(L.g, 0.0f);
            L.gU = array(L.g, 0.0f);
            L.finv = array(L.g, 0.5f);
            L.x = array(L.g, 3.0f);
            L.b = array(L.g, 1.0f);
            v.push_back(L);
            if (nx == 1 && ny == 1) break;
            nx = (nx + 1) / 2, ny = (ny + 1) / 2;
        }
    }
    ~Stack() {
        for (float* d : owned) cudaFree(d);
    }
};

int launch(const TailPlan& p, const Stack& s, const std::vector<int>& table) {
    TailMaps m;
    if (!make_tail_maps(p, s.v.data(), &m)) return 1;
    int* dt = nullptr;
    Ctl *dc = nullptr, c;
    std::memset(&c, 0, sizeof c);
    const size_t n = (size_t)s.v[0].g.plane * s.v[0].g.nz;
    std::vector<float> before(n), after(n);
    if (cudaMalloc(&dt, table.size() * 4) != cudaSuccess || cudaMalloc(&dc, sizeof c) != cudaSuccess) return 1;
    cudaMemcpy(dt, table.data(), table.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(dc, &c, sizeof c, cudaMemcpyHostToDevice);
    cudaMemcpy(before.data(), s.v[0].x, n * 4, cudaMemcpyDeviceToHost);
    if (launch_tail(nullptr, p, m, dt, dc, Cond{0, 0}) != cudaSuccess) return 1;
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    cudaMemcpy(&c, dc, sizeof c, cudaMemcpyDeviceToHost);
    cudaMemcpy(after.data(), s.v[0].x, n * 4, cudaMemcpyDeviceToHost);
    std::printf("launch %d %d %d %d %d\n", p.ctas, c.err, c.breakdown, c.done, before == after ? 0 : 1);
    cudaFree(dt);
    cudaFree(dc);
    return 0;
}
}  // namespace

int main() {
    int devices = 0;
    if (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0) return 3;
    // a cluster with the bottom levels on a CTA of their own, one with the first
    // rows' CTA holding them, and one CTA alone
    const int sizes[3][2] = {{64, 64}, {64, 64}, {13, 11}};
    for (int k = 0; k < 3; ++k) {
        Stack s(sizes[k][0], sizes[k][1], 10);
        TailPlan p;
        if (!plan_tail(s.v.data(), (int)s.v.size(), kTailCtas, k == 0, kTailSmemMax, &p)) return 1;
        std::vector<int> table((size_t)p.table_bytes / 4);
        fill_tail_table(p, table.data());
        TailPlan late = p;
        late.polls = 20000;
        late.first_bytes += 16;
        late.bottom_first_bytes += 16;
        late.dist_bytes += 16;
        late.bottom_bytes += 16;
        if (launch(late, s, std::vector<int>(table.size(), 0x7fffffff))) return 1;
        if (launch(p, s, table)) return 1;
    }
    return 0;
}
