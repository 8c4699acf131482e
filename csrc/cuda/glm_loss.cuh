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
