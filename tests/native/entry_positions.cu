// Loops over a row's entries where the row ends at the largest entry count a
// graph may have (2^31 - 1): they visit the row's entries and stop.
#include "../../acc-gp_b200/csrc/gp_graph.h"
#include "fake_runtime.h"

using namespace gp;

// The form of the kernels' loops: entries first, first + stride, ... < end, U at a time.
static void walk(int row_begin, int row_end, u32 lane, u32 stride, u32 U) {
    EXPECT(U * stride <= kEntryStep);
    const EntryPos begin = row_begin, end = row_end;
    i64 visits = 0, steps = 0;
    for (EntryPos e0 = begin + lane; e0 < end; e0 += U * stride) {
        EXPECT(++steps < (i64{1} << 20));
        for (u32 j = 0; j < U; ++j) {
            const EntryPos e = e0 + j * stride;
            if (e >= end) continue;
            EXPECT(static_cast<i64>(e) >= row_begin && static_cast<i64>(e) < row_end);
            ++visits;
        }
    }
    const i64 length = static_cast<i64>(row_end) - row_begin;
    EXPECT(visits == (length > lane ? (length - lane + stride - 1) / stride : 0));
}

int main() {
    const int top = 0x7fffffff;
    for (int end : {top, top - 1, top - 2047, top - 4096, 5000})
        for (int length : {0, 1, 5, 31, 2048, 2049, 4990})
            for (u32 lane : {0u, 1u, 31u})
                for (u32 stride : {1u, 8u, 32u, 256u}) {
                    walk(end - length, end, lane, stride, 1);
                    walk(end - length, end, lane, stride, 4);
                    walk(end - length, end, lane, stride, 8);
                }
    walk(0, 0, 1023, 1024, 4);
    walk(top - 9000, top, 1023, 1024, 4);

    for (int size : {256, 2048}) {
        EXPECT(row_pieces(0, size) == 0 && row_pieces(1, size) == 1 && row_pieces(size, size) == 1);
        EXPECT(row_pieces(size + 1, size) == 2);
        EXPECT(row_pieces(top, size) == (i64{top} + size - 1) / size);
        EXPECT(row_pieces(top - size + 2, size) == (i64{top} - size + 2 + size - 1) / size);
    }

    // The last chunk of a row that ends at the top, begun within a chunk of it.
    int off[2] = {top - 5000, top};
    int chunk_begin[3] = {top - 5000, top - 5000 + kChunk, top - 5000 + 2 * kChunk};
    DGraph g;
    g.off = off;
    g.chunk_begin = chunk_begin;
    EXPECT(chunk_end(g, 0, 0) == static_cast<EntryPos>(chunk_begin[1]));
    EXPECT(chunk_end(g, 1, 0) == static_cast<EntryPos>(chunk_begin[2]));
    EXPECT(chunk_end(g, 2, 0) == static_cast<EntryPos>(top));
    return 0;
}
