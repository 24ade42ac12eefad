// Host view of the batched sweeps' tile counts (sweep_dispatch.h) for
// tests/test_batch_tiling_host.py.
#include "sweep_dispatch.h"

extern "C" long long h_batch_tiles(int nv, int ax, int nx, int ny, int nz, int seg_len, int prec, int shape)
{
    cfd::SweepParams p = {};
    p.n[0] = nx;
    p.n[1] = ny;
    p.n[2] = nz;
    p.seg_len = seg_len;
    p.prec = prec;
    return cfd::sweep_tile_count(nv, ax, p, shape);
}
