// CPU check of how a layer call cuts its rows: the windows cover the promised rows (or the whole capacity) once, the chunks of
// a window begin at whole minibatches and stay bounded in number, and with several ranks they are the fixed size that was
// measured there.  Built and run by tests/test_layer_windows.py.
#include <cstdio>
#include <initializer_list>

#include "../mixture-of-kittens_b200/csrc/layer_windows.cuh"

using namespace mok;

#define CHECK(cond)                                                                                                          \
    do {                                                                                                                     \
        if (!(cond)) {                                                                                                       \
            std::printf("FAILED %s: ep %d capacity %d promised %d ring %d window %d chunk %d\n", #cond, ep, cap, promised, ring, rows, \
                        chunk);                                                                                              \
            return 1;                                                                                                        \
        }                                                                                                                    \
    } while (0)

int main() {
    for (int ep : {1, 2, 8})
        for (int mini : {256, 4096})
            for (int ring : {mini, 3 * mini, 32 * mini, 120 * mini})
                for (int cap : {256, 49152, 49408, 262144, 524288})
                    for (int promised : {0, 256, 40192, 270336}) {
                        mok_layer_args a{};
                        a.ep_size = ep;
                        a.minibatch_size = mini;
                        a.macrobatch_size = ring;
                        a.schedule_capacity = cap;
                        a.schedule_rows = promised;
                        int rows = 0, chunk = 0, next = 0;
                        for (int w = 0; w < num_windows(&a); ++w) {
                            const Span s = window_span(&a, w);
                            rows = s.end - s.begin;
                            CHECK(s.begin == next && s.base == s.begin && rows > 0 && rows <= ring);
                            next = s.end;
                            chunk = chunk_rows_for(&a, rows, false);
                            const int n = (rows + chunk - 1) / chunk, fixed = kMinibatchesPerChunk * mini;
                            CHECK(chunk > 0 && chunk <= rows && n <= 101 && (n == 1 || chunk % mini == 0));
                            if (ep > 1 && ring <= 100 * fixed) CHECK(chunk == (fixed < rows ? fixed : rows));
                            if (ep == 1) CHECK(n > 1 || 2 * rows < 3 * fixed);
                            CHECK(ep > 1 || chunk_rows_for(&a, rows, true) == rows);
                        }
                        CHECK(next == (promised > 0 && promised < cap ? promised : cap));
                    }
    std::printf("ok\n");
    return 0;
}
