// The skew fallback's error exit, on hand-made state: with a device error
// noted before its first barrier, every member leaves without touching the
// batch, the last one copies the counters and leaves them and the gate clean.
// Without the gate's flag the launch changes nothing.
#include <chrono>
#include <stdio.h>
#include <string.h>

#include "../../ltpmg_gb300/csrc/ltp_internal.cuh"

using namespace ltp;

struct State {
    PartState st;
    Counters ctr, snap;
};

int main() {
    State *s;
    Launch L;
    int dev = 0;
    memset(&L, 0, sizeof(L));
    if (cudaMallocManaged(&s, sizeof(State)) != cudaSuccess) return 2;
    if (cudaDeviceGetAttribute(&L.num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 2;
    if (cudaStreamCreate(&L.stream) != cudaSuccess) return 2;
    BatchDev b;
    TablesDev T;
    Scratch sc;
    memset(&b, 0, sizeof(b));  // no transaction, no op
    memset(&T, 0, sizeof(T));
    memset(&sc, 0, sizeof(sc));
    sc.pstate = &s->st;
    sc.fctr = &s->ctr;
    for (int k = 0; k < 200; k++) {
        const bool skew = k % 4 != 3;
        memset(s, 0, sizeof(*s));
        s->st.skew = skew;
        s->ctr.err = LTP_E_DEVICE_ASSERT;
        s->ctr.n_c = 41;
        const auto t0 = std::chrono::steady_clock::now();
        if (launch_fallback(L, b, T, sc, &s->snap) != cudaSuccess || cudaStreamSynchronize(L.stream) != cudaSuccess) return 2;
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        bool ok = s->st.skew == 0 && ms < 1000;
        if (skew)
            ok = ok && s->snap.err == LTP_E_DEVICE_ASSERT && s->snap.n_c == 41 && s->ctr.err == 0 && s->ctr.n_c == 0 &&
                 s->st.members >= 1 && s->st.left == s->st.members;
        else
            ok = ok && s->snap.err == 0 && s->ctr.err == LTP_E_DEVICE_ASSERT && s->ctr.n_c == 41 && s->st.joined == 0;
        if (!ok) {
            printf("launch %d: skew %u snapshot %d counters %d members %u left %u, %.1f ms\n", k, s->st.skew, s->snap.err,
                   s->ctr.err, s->st.members, s->st.left, ms);
            return 1;
        }
    }
    puts("ok");
    return 0;
}
