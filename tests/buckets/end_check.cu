// The kernel that closes a bucket batch with inserts, on hand-made state: a
// device error noted after the snapshot was taken (by the row kernel of a
// bounds-checked build) reaches the snapshot, and the row counts stay.
#include "../../ltpmg_gb300/csrc/ltp_buckets.cu"

#include <stdio.h>

using namespace ltp;

struct State {
    PartState st;
    PartCounters ctr[2];
    Counters snap;
    u64 rows[LTP_MAX_TABLES];
    u32 ins_pre[2 * LTP_MAX_TABLES];
};

int main() {
    State *s;
    if (cudaMallocManaged(&s, sizeof(State)) != cudaSuccess) return 2;
    struct { int err, snapped; u32 full; int want; u64 rows; } cases[] = {
        {0, 0, 0, 0, 107},                                       // all well: 7 rows more
        {LTP_E_DEVICE_ASSERT, 0, 0, LTP_E_DEVICE_ASSERT, 100},   // noted late
        {LTP_E_BADARG, LTP_E_BADARG, 0, LTP_E_BADARG, 100},      // known before
        {0, LTP_E_CAPACITY, 1, LTP_E_CAPACITY, 100},             // refused for want of room
        {LTP_E_DEVICE_ASSERT, LTP_E_CAPACITY, 0, LTP_E_CAPACITY, 100},  // the first error stays
    };
    for (u32 par = 0; par < 2; par++)
        for (auto &c : cases) {
            memset(s, 0, sizeof(*s));
            s->st.par2 = par;
            s->st.full = c.full;
            s->ctr[par].c.err = c.err;
            s->ctr[par].c.ins_committed[1] = 7;
            s->ctr[par ^ 1].c.err = LTP_E_TIMEOUT;  // (another batch's)
            s->snap.err = c.snapped;
            s->rows[1] = 100;
            for (u32 &x : s->ins_pre) x = 9;
            BatchDev b;
            TablesDev T;
            BucketPlan p;
            memset(&b, 0, sizeof(b));
            memset(&T, 0, sizeof(T));
            memset(&p, 0, sizeof(p));
            b.n_ops = kInsTile + 1;
            T.n = 2;
            T.rows_now = s->rows;
            p.state = &s->st;
            p.ctr = s->ctr;
            p.snap = &s->snap;
            p.ins_pre = s->ins_pre;
            k_end<<<1, 1024>>>(b, T, p);
            if (cudaDeviceSynchronize() != cudaSuccess) return 2;
            bool ok = s->snap.err == c.want && s->rows[1] == c.rows && s->rows[0] == 0 && s->st.full == 0;
            for (u32 x : s->ins_pre) ok = ok && x == 0;
            if (!ok) {
                printf("err %d, snapshot %d: snapshot %d, rows %llu\n", c.err, c.snapped, s->snap.err, s->rows[1]);
                return 1;
            }
        }
    puts("ok");
    return 0;
}
