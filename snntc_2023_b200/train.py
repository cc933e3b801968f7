"""What surrounds the SNN-TC layers in a training step of the reference's example trainers, on this
library's own kernels (csrc/snntc_train.cu) instead of framework glue:

    encode(p)                       exp(1 - p) / exp(p) input encoding            snntc-mnist.py:75
    loss_func(logit, label)         softmax cross-entropy on -logit, batch mean   SNN_TC_Modules.py:286-288
    accuracy_count(logit, label)    number of samples whose earliest spike is the label   snntc-mnist.py:82
    constraint_cost(weights, K, K2) K*sum_w mean_j max(0,1-sum_i w_ij) + K2*sum_w mean(w^2)   snntc-mnist.py:55-59
    Adam / SGDM                     Keras-formulation optimisers over one flat parameter buffer and the
                                    flat gradient buffer the backward kernels (and the all-reduce) write

Everything here needs the CUDA library; there is no CPU path.
"""

import torch

from . import _lib
from .ops import _as_cuda_f32, _stream, _tensor


def encode(p, scale=1.0, one_minus=True):
    """x = exp(scale*(1-p)) (pixel intensities -> spike times, the reference's encoding) or exp(scale*p)."""
    return _lib.native().encode(_tensor(p, "p"), scale, one_minus)


def loss_func(logit=None, label=None, with_hits=False):
    """Mean softmax cross-entropy on the negated spike times. `label`: integer classes [B] or one-hot [B,C].
    with_hits=True also returns the number of samples whose arg-min output equals the label (a 0-d tensor)."""
    loss, hits = _lib.native().loss(_tensor(logit, "logit"), label)
    return (loss, hits) if with_hits else loss


def accuracy_count(logit, label):
    with torch.no_grad():
        return loss_func(logit, label, with_hits=True)[1]


def constraint_cost(weights, K, K2):
    """K * sum over tensors of mean_j max(0, 1 - sum_i w_ij) + K2 * sum over tensors of mean(w^2); each tensor is
    a layer's whole [fan_in(+1), fan_out] weight, bias row included, as in the reference's trainable_variables."""
    return _lib.native().constraint_cost(list(weights), K, K2)


class _FlatOptimizer:
    def __init__(self, param, grad):
        self.param = _as_cuda_f32(param.detach() if isinstance(param, torch.nn.Parameter) else param, "param")
        self.grad = _as_cuda_f32(grad, "grad")
        if self.param.numel() != self.grad.numel():
            raise ValueError("parameter and gradient buffers differ in size")

    def zero_grad(self):
        self.grad.zero_()


class Adam(_FlatOptimizer):
    """tf.keras.optimizers.Adam over one flat fp32 buffer; the step count lives on the device, so step() can be
    captured into a CUDA graph and replayed. grad_scale multiplies the gradient first (1/world for a summed
    all-reduce)."""

    def __init__(self, param, grad, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-7):
        super().__init__(param, grad)
        self.lr, self.beta1, self.beta2, self.eps = lr, beta1, beta2, eps
        self.m = torch.zeros_like(self.param)
        self.v = torch.zeros_like(self.param)
        self.steps = torch.zeros(1, dtype=torch.int32, device=self.param.device)

    def step(self, grad_scale=1.0):
        _lib.native().adam_step(self.param, self.grad, self.m, self.v, self.lr, self.beta1, self.beta2, self.eps,
                                grad_scale, self.steps)


class SGDM(_FlatOptimizer):
    """tf.keras.optimizers.SGD(momentum=...): vel = momentum*vel - lr*g; w += vel."""

    def __init__(self, param, grad, lr=1e-2, momentum=0.9):
        super().__init__(param, grad)
        self.lr, self.momentum = lr, momentum
        self.vel = torch.zeros_like(self.param)

    def step(self, grad_scale=1.0):
        lib = _lib.load()
        with torch.cuda.device(self.param.device):
            rc = lib.snntc_sgdm_step(self.param.data_ptr(), self.grad.data_ptr(), self.vel.data_ptr(),
                                     self.param.numel(), float(self.lr), float(self.momentum), float(grad_scale),
                                     _stream(self.param))
        _lib.check(rc, "SGDM.step")
