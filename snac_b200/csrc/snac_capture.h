// snac_capture.h — records launches into an executable graph (plain C++, so
// that the host can check what a failure leaves behind).
//
// Api: the CUDA calls and the caller's bookkeeping:
//   int begin(), end(Graph*), instantiate(Exec*, Graph); void destroy(Graph)
//   Mark mark(), void restore(Mark), long long launched_since(Mark)
// Each int is a status, 0 for success.
#pragma once

namespace snac {

// Records what record() launches.  The bookkeeping that recording advances (launches,
// time step, coordinate buffer) is afterwards what it was: the kernels run,
// and count, when the graph is launched.  On a failure of any call the stream
// has left the capture, the graph is destroyed and *out keeps its value.
template <class Api, class Record>
int capture_graph(Api& api, Record record, typename Api::Exec* out, int* kernels) {
    const auto before = api.mark();
    int rc = api.begin();
    if (rc) return rc;
    rc = record();
    typename Api::Graph g{};
    const int ended = api.end(&g);
    const int launched = (int)api.launched_since(before);
    api.restore(before);
    if (!rc) rc = ended;
    typename Api::Exec e{};
    if (!rc) rc = api.instantiate(&e, g);
    if (g) api.destroy(g);
    if (rc) return rc;
    *out = e;
    *kernels = launched;
    return 0;
}

}  // namespace snac
