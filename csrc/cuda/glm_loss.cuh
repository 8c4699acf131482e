// Loss and negative derivative of the three linear models (objective/Loss.scala:82-137 of the reference's ml module:
// log, hinge and square loss, +-18 cut-offs).
#pragma once
#include <math.h>

__device__ __forceinline__ float glm_loss(int loss_id, float pre, float y) {
    if (loss_id == 0) {
        float z = pre * y;
        if (z > 18.f) return __expf(-z);
        if (z < -18.f) return -z;
        return log1pf(__expf(-z));
    } else if (loss_id == 1) {
        float z = pre * y;
        return z < 1.f ? 1.f - z : 0.f;
    }
    float d = pre - y;
    return 0.5f * d * d;
}

// negative derivative of the loss with respect to the prediction
__device__ __forceinline__ float glm_grad(int loss_id, float pre, float y) {
    if (loss_id == 0) {
        float z = pre * y;
        if (z > 18.f) return y * __expf(-z);
        if (z < -18.f) return y;
        return y / (1.f + __expf(z));
    } else if (loss_id == 1) {
        return pre * y <= 1.f ? y : 0.f;
    }
    return y - pre;
}

// The loss partials of a step, {rows, loss sum, regularisation, -}: the gradient kernels add the loss to the spare word
// of the template that holds the rest, and a kernel behind them puts both together for the step and clears the word, so
// that neither needs a launch (a copy of 32 bytes cost 1.5 us and the gap before the next kernel 2 us).
struct StepLoss {
    double* partials;   // null: the caller sees to it
    double* tmpl;
    __device__ __forceinline__ void settle() const {
        if (!partials) return;
        partials[0] = tmpl[0];
        partials[1] = tmpl[1] + tmpl[3];
        partials[2] = tmpl[2];
        partials[3] = 0.0;
        tmpl[3] = 0.0;
    }
};
