// capture_graph with each of its calls failing in turn: the stream has left the
// capture, no graph is left over, the bookkeeping is what it was.
#include <cstdio>

#include "snac_capture.h"

namespace {

struct Fake {
    using Graph = int;
    using Exec = int;
    struct Mark {
        long long launches, time_step;
        int parity;
    };
    int fail = 0;  // 1 begin, 2 end, 3 instantiate; 4 the recording, at its second step
    bool capturing = false;
    int graphs = 0;
    Mark state{7, 40, 1};
    Mark mark() const { return state; }
    void restore(Mark m) { state = m; }
    long long launched_since(Mark m) const { return state.launches - m.launches; }
    int begin() {
        if (fail == 1) return -1;
        capturing = true;
        return 0;
    }
    int end(Graph* g) {
        capturing = false;
        if (fail == 2) return -2;  // (a capture that was invalidated gives no graph)
        graphs++;
        *g = 5;
        return 0;
    }
    int instantiate(Exec* e, Graph) {
        if (fail == 3) return -3;
        *e = 9;
        return 0;
    }
    void destroy(Graph) { graphs--; }
};

}  // namespace

int main() {
    int bad = 0;
    for (int fail = 0; fail <= 4; fail++) {
        Fake f;
        f.fail = fail;
        int exec = -1, kernels = -1;
        const int rc = snac::capture_graph(
            f,
            [&] {
                for (int s = 0; s < 3; s++) {  // an odd number of steps: the buffers change places
                    if (fail == 4 && s == 1) return -4;
                    f.state.launches += 3;
                    f.state.time_step++;
                    f.state.parity ^= 1;
                }
                return 0;
            },
            &exec, &kernels);
        bad += rc != -fail;
        bad += f.capturing;
        bad += f.graphs != 0;
        bad += f.state.launches != 7 || f.state.time_step != 40 || f.state.parity != 1;
        bad += fail ? exec != -1 || kernels != -1 : exec != 9 || kernels != 9;
    }
    if (bad) printf("%d checks failed\n", bad);
    return bad != 0;
}
