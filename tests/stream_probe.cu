// Prints the dispatch rule of the streaming matvec: one line per question read from standard input.
//   pass <qtype> <rows> <width> <count> <matrix_stride> <has matrix_ptrs> <has x_rows> <has activation>   -> input rows per pass
#include <cstdio>

#include "gemv_stream.cuh"

int main() {
    unsigned q;
    unsigned long long matrix_rows, width, count, stride;
    int ptrs, rows, act;
    while (scanf(" pass %u %llu %llu %llu %llu %d %d %d", &q, &matrix_rows, &width, &count, &stride, &ptrs, &rows, &act) == 8) {
        const yb::Geometry g = yb::geometry_of(q);
        yb::gs::StreamShape sh{};
        const uint8_t *const some_ptrs[1] = {nullptr};
        const uint32_t some_rows[1] = {0};
        const yb::gs::StreamActivation some_act{nullptr, nullptr, 0.0f};
        printf("%d\n", yb::gs::pass_inputs(q, matrix_rows, width, width / g.elems * g.bytes, count, stride, ptrs ? some_ptrs : nullptr, rows ? some_rows : nullptr,
                                           act ? &some_act : nullptr, sh));
    }
    return 0;
}
