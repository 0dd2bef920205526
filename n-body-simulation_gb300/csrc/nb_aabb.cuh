// nb_aabb.cuh -- device parts of the AABB shared by nb_integrate.cu and the one-block octree build:
// order-preserving integer images of doubles and the reference's cube rule.
#pragma once

namespace nbaabb {

__device__ __forceinline__ long long ord_of(double v) {
    const long long b = __double_as_longlong(v);
    return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double val_of(long long o) {
    return __longlong_as_double(o >= 0 ? o : (o ^ 0x7fffffffffffffffLL));
}

struct MinMax6 {
    long long v[6];  // min x, y, z (as ordered ints), max x, y, z
};

__device__ inline void cube_rule(double min_x, double min_y, double min_z, double max_x, double max_y,
                          double max_z, double* out) {
    const double x_len = fabs(__dsub_rn(max_x, min_x));
    const double y_len = fabs(__dsub_rn(max_y, min_y));
    const double z_len = fabs(__dsub_rn(max_z, min_z));
    const double edge = fmax(x_len, fmax(y_len, z_len));
    if (edge == x_len) {
        min_z = __dsub_rn(min_z, __dsub_rn(edge, z_len) / 2);
        min_y = __dsub_rn(min_y, __dsub_rn(edge, y_len) / 2);
        max_z = __dadd_rn(max_z, __dsub_rn(edge, z_len) / 2);
        max_y = __dadd_rn(max_y, __dsub_rn(edge, y_len) / 2);
    } else if (edge == y_len) {
        min_x = __dsub_rn(min_x, __dsub_rn(edge, x_len) / 2);
        min_z = __dsub_rn(min_z, __dsub_rn(edge, z_len) / 2);
        max_x = __dadd_rn(max_x, __dsub_rn(edge, x_len) / 2);
        max_z = __dadd_rn(max_z, __dsub_rn(edge, z_len) / 2);
    } else {
        min_x = __dsub_rn(min_x, __dsub_rn(edge, x_len) / 2);
        min_y = __dsub_rn(min_y, __dsub_rn(edge, y_len) / 2);
        max_x = __dadd_rn(max_x, __dsub_rn(edge, x_len) / 2);
        max_y = __dadd_rn(max_y, __dsub_rn(edge, y_len) / 2);
    }
    out[0] = min_x;
    out[1] = min_y;
    out[2] = min_z;
    out[3] = max_x;
    out[4] = max_y;
    out[5] = max_z;
    out[6] = edge;
}

}  // namespace nbaabb
