// Host memory running out while the tiles are built (test infrastructure): every allocation in turn fails
// once, on whichever thread makes it, and the builder has to report MEL_ERR_OOM instead of ending the
// process.  Arguments: bodies, points a body, supports a point.  Prints how often each call reported
// it; exits 0 when all went as it should.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include "mel_tiles.h"

static std::atomic<long long> g_left{ -1 };       // allocations until the one that fails; -1: none does

void* operator new(size_t n)
{
    if (g_left.load() >= 0 && g_left.fetch_sub(1) == 0) throw std::bad_alloc();
    void* p = malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

void mel_set_error(const char*, ...) {}

int main(int, char** argv)
{
    const int nb = atoi(argv[1]), np = atoi(argv[2]), ns = atoi(argv[3]), nn = 4 * ns;
    std::vector<int> type(nb, MEL_BODY_DEFORMABLE), nptr(nb + 1), gptr(nb + 1), sptr(nb * np + 1), idx((size_t)nb * np * ns);
    std::vector<double> v(idx.size(), 1.), w((size_t)nb * np, 1.);
    for (int b = 0; b <= nb; b++) { nptr[b] = b * nn; gptr[b] = b * np; }
    for (size_t g = 0; g < sptr.size(); g++) sptr[g] = (int)g * ns;
    for (size_t e = 0; e < idx.size(); e++) idx[e] = (int)((e * 7 + e / ns) % nn);
    mel_model_desc d;
    memset(&d, 0, sizeof d);
    d.n_bodies = nb; d.n_nodes = nb * nn; d.n_gauss = nb * np;
    d.body_type = type.data(); d.body_node_ptr = nptr.data(); d.body_gp_ptr = gptr.data(); d.gp_sup_ptr = sptr.data();
    d.gp_sup_idx = idx.data(); d.gp_dNdx = v.data(); d.gp_dNdy = v.data(); d.gp_weight = w.data(); d.gp_jacobian = w.data();
    int plan_oom = 0, fill_oom = 0, fine = 0;
    for (long long k = 0; k < 4000; k += 1 + k / 20) {
        mel_tile_set TS;
        g_left = k;
        int rc = mel_plan_tiles(&d, 3840, false, TS);
        g_left = -1;
        if (rc == MEL_ERR_OOM) { plan_oom++; if (mel_plan_tiles(&d, 3840, false, TS) != MEL_OK) return 2; }
        else if (rc != MEL_OK) return 3;
        g_left = k;
        rc = mel_fill_tiles(&d, TS);
        g_left = -1;
        if (rc == MEL_ERR_OOM) fill_oom++;
        else if (rc == MEL_OK) fine++;
        else return 4;
    }
    printf("%d %d %d\n", plan_oom, fill_oom, fine);
    return 0;
}
