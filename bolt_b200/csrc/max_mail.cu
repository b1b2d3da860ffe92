// max_mail.cu -- the pool of MaxMails: who may use one, when it is free again, and the host's wait for its report.
#include <sched.h>

#include "common.cuh"

namespace b200 {

MaxLease::MaxLease(DeviceCtx *c) : c_(c)
{
    std::unique_lock<std::mutex> g(c->mail_mu);
    c->mail_cv.wait(g, [&] { return !c->mail_free.empty() || c->mails == 0; });
    if (c->mail_free.empty()) {
        return;   // none is left: the device has failed before
    }
    m_ = c->mail_free.back();
    c->mail_free.pop_back();
    if (++m_->seq == 0) {
        m_->seq = 1;
    }
}

// A mail whose kernel has not been seen to report may still be in that kernel's hands, and its words may be half
// counted: it goes back only behind the end of the stream's work and with its words rewound, or not at all.
MaxLease::~MaxLease()
{
    if (m_ == nullptr) {
        return;
    }
    const bool usable = !in_flight_ || (cudaStreamSynchronize(st_) == cudaSuccess && cudaMemsetAsync(m_->words, 0, 8, st_) == cudaSuccess &&
        cudaStreamSynchronize(st_) == cudaSuccess);
    if (!usable) {
        cudaGetLastError();
    }
    {
        std::lock_guard<std::mutex> g(c_->mail_mu);
        if (usable) {
            c_->mail_free.push_back(m_);
        } else {
            --c_->mails;
        }
    }
    c_->mail_cv.notify_all();   // (a waiter also has to learn that the last mail is gone)
}

EE MaxLease::wait(int *maximum)
{
    auto arrived = [&] {
        const unsigned long long v = *m_->h_mail;
        *maximum = (int)(unsigned)v;
        return (uint32_t)(v >> 32) == m_->seq;
    };
    for (uint32_t spin = 1;; ++spin) {
        if (arrived()) {
            in_flight_ = false;   // (the report is the last that the kernel does with its mail)
            return SUCCESS;
        }
        __builtin_ia32_pause();
        if ((spin & 0x3FFF) == 0) {   // some hundred microseconds: is the stream still at work?
            const cudaError_t e = cudaStreamQuery(st_);
            if (e == cudaErrorNotReady) {
                cudaGetLastError();
                sched_yield();
                continue;
            }
            if (e == cudaSuccess && arrived()) {
                in_flight_ = false;
                return SUCCESS;
            }
            return e == cudaSuccess ? UNKNOWN : cuda_ee(e);
        }
    }
}

bool capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) != cudaSuccess) {
        cudaGetLastError();
        return true;   // the legacy stream beside another stream's capture
    }
    return s != cudaStreamCaptureStatusNone;
}

}  // namespace b200
