// The pool of MaxMails against a fake CUDA runtime (fake_cudart.cpp, linked instead of the real one): what happens to a mail whose kernel
// has not reported, on the CPU.  Prints "ok", or the first condition that does not hold.
#include <cstdio>
#include <cstdlib>

#include "common.cuh"

using namespace b200;

extern int (*on_query)(void);          // fake_cudart.cpp
extern int (*on_synchronize)(void);

namespace b200 {
EE cuda_ee(cudaError_t e)
{
    return e == cudaSuccess ? SUCCESS : UNKNOWN;
}
}  // namespace b200

namespace {

struct Fake {
    cudaError_t query = cudaErrorNotReady, sync = cudaSuccess;   // what the calls answer
    int queries = 0, syncs = 0;
    int report_after = -1;                  // the kernel reports at this query
    bool free_at_sync = false;              // a mail of the running kernel was in the pool while the stream was waited for
    const MaxMail *mail = nullptr;          // of the kernel in flight
    int value = 0;
} fake;
DeviceCtx *pool = nullptr;

int query()
{
    if (++fake.queries == fake.report_after) {
        const unsigned long long v = ((unsigned long long)fake.mail->seq << 32) | (unsigned)fake.value;
        *fake.mail->h_mail = v;
    }
    return fake.query;
}
int synchronize()
{
    ++fake.syncs;
    for (const MaxMail *m : pool->mail_free) {
        fake.free_at_sync |= m == fake.mail;
    }
    return fake.sync;
}
#define HOLDS(cond)                                                        \
    do {                                                                   \
        if (!(cond)) {                                                     \
            std::printf("%s:%d: %s\n", __func__, __LINE__, #cond);         \
            std::exit(1);                                                  \
        }                                                                  \
    } while (0)

DeviceCtx *make_pool(int n)
{
    DeviceCtx *c = new DeviceCtx();
    for (int i = 0; i < n; ++i) {
        MaxMail *m = new MaxMail();
        m->words = new unsigned[8]();
        m->d_mail = nullptr;
        m->h_mail = new unsigned long long[8]();
        m->seq = 0;
        c->mail_free.push_back(m);
    }
    c->mails = n;
    fake = Fake();
    return pool = c;
}

void reports_while_polled()
{
    DeviceCtx *c = make_pool(1);
    for (int round = 0; round < 3; ++round) {
        MaxLease l(c);
        HOLDS(l.ok());
        fake.mail = &l.mail();
        fake.value = 100 + round;
        fake.report_after = fake.queries + 2;
        l.launched(nullptr);
        int mx = 0;
        HOLDS(l.wait(&mx) == SUCCESS && mx == 100 + round);
    }
    HOLDS(fake.syncs == 0 && c->mail_free.size() == 1);
}
void not_launched()
{
    DeviceCtx *c = make_pool(1);
    {
        MaxLease l(c);
    }
    HOLDS(fake.syncs == 0 && c->mail_free.size() == 1);
}
// an error between the launch and the wait
void left_in_flight()
{
    DeviceCtx *c = make_pool(2);
    unsigned *words = nullptr;
    {
        MaxLease l(c);
        fake.mail = &l.mail();
        words = l.mail().words;
        words[0] = 77;      // the kernel has begun to count
        words[1] = 3;
        l.launched(nullptr);
    }
    HOLDS(fake.syncs >= 1 && !fake.free_at_sync);
    HOLDS(words[0] == 0 && words[1] == 0 && c->mail_free.size() == 2 && c->mails == 2);
}
void ends_without_a_report()
{
    DeviceCtx *c = make_pool(1);
    for (int round = 0; round < 100; ++round) {
        MaxLease l(c);
        HOLDS(l.ok());
        fake.mail = &l.mail();
        fake.query = cudaSuccess;
        l.mail().words[1] = 5;
        l.launched(nullptr);
        int mx = 0;
        HOLDS(l.wait(&mx) == UNKNOWN);
    }
    HOLDS(c->mail_free.size() == 1 && c->mail_free[0]->words[1] == 0);
}
// the device has failed: every call returns an error, none waits for a mail that will not come back
void device_gone()
{
    DeviceCtx *c = make_pool(3);
    fake.query = fake.sync = cudaErrorLaunchFailure;
    for (int round = 0; round < 3; ++round) {
        MaxLease l(c);
        HOLDS(l.ok());
        fake.mail = &l.mail();
        l.launched(nullptr);
        int mx = 0;
        HOLDS(l.wait(&mx) != SUCCESS);
    }
    MaxLease l(c);
    HOLDS(!l.ok());
}

}  // namespace

int main()
{
    on_query = query;
    on_synchronize = synchronize;
    reports_while_polled();
    not_launched();
    left_in_flight();
    ends_without_a_report();
    device_gone();
    std::puts("ok");
    return 0;
}
