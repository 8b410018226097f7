// Host build of axis_cut for tests/test_axis_cut.py: polygons in, polygons out.
#include "geom2d.cuh"

extern "C" int axis_cut_host(double *x, double *y, int *id, int m, int cap, int axis, double c, double s, int own, int room) {
    const sdot::PolyView<double> q{x, y, id, 1, cap};
    return sdot::axis_cut(q, m, axis, c, s, own, room);
}
