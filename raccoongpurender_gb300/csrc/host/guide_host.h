// guide_host.h — the host object behind rgr_guide: the path-guiding network
// and its optimiser state on one device, plus the training-sample stream a
// guided render feeds.
#pragma once
#include "../kernels/guide.cuh"
#include "devbuf.h"
#include "mail.h"

struct rgr_guide {
    int device = 0;
    int num_sms = 152;
    rgr_guide_config cfg{};
    // network: FP32 master weights and biases, BF16 weights, gradients, Adam moments, loss
    rgr::DevBuf w, b, wbf, gW, gb, m, v, loss;
    // training stream: samples, counters, loss history
    rgr::DevBuf samples, counters, loss_hist, wtsw;
    rgr::DevBuf gpart;  // the tcgen05 training kernel's per-CTA gradient slots (num_sms x kGuidePartStride)
    rgr::dev::GuideView view{};
    rgr::dev::GuideTrainD train{};  // the render's stream (counter bytes 0..27)
    rgr::dev::GuideTrainD test{};   // rgr_guide_train_device's (bytes 32..59; shares iter)
    bool bounds_set = false;
    rgr::MailSlot mail;  // the last training step's loss

    int init(const rgr_guide_config& c);
    int set_bounds(const float lo[3], const float hi[3]);
    // the bounce's inference launch (tcgen05 or mma.sync kernel, per cfg)
    // inner: the render's request, for a bounce inside a run (launch_inner_queues); else null
    void infer_paths(const rgr::dev::PathsView& p, const rgr::dev::QueueView& q, const rgr::dev::GuideRenderD& gd,
                     const rgr::dev::RequestD* inner, cudaStream_t st);
    // renders with the weights as they are: such a render's bounces need no logic pass of their own
    bool frozen() const { return !cfg.train && cfg.inference_kernel == RGR_GUIDE_TCGEN05; }
    uint32_t* error_word() const;
    // the launches that follow the trace/logic kernel of a guided render on the
    // bounces that end a training interval: train, Adam, reset the stream
    int train_launches(cudaStream_t st);
    rgr::dev::GuideAdam adam() const;
    // one iteration with the tcgen05 kernels over min(*count, n) samples (n with count null):
    // gradients to `grads` if given; with `step`, Adam and the bookkeeping of t; `grid` CTAs
    void iteration_launches(const float* samples, const uint32_t* count, uint32_t n, const rgr::dev::GuideTrainD& t,
                            const float* wsum, float weight_scale, int grid, bool step, float* grads, float* host_loss,
                            cudaStream_t st);
};
