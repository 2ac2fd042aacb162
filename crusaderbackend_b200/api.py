"""Thin Python face of the C ABI for tests and benchmarks.

torch is used only to own device memory and streams; every computation goes through
libcrusader_b200.so, called by the extension module _native (csrc/bind.cpp), which reads the tensors'
extents, strides and pointers natively. Function names follow the reference's seblas operations
(seblas/operations/cuGEMM.cuh:12-21, cuConv.cuh:20-42, cuLinear.cuh:14-18).
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from ._lib import CB_MATH_3XTF32, CB_MATH_FP32, CB_MATH_TF32, CrusaderError

MATH_MODES = {"tf32": CB_MATH_TF32, "3xtf32": CB_MATH_3XTF32, "fp32": CB_MATH_FP32}


_native = None


def _load_native(lib: C.CDLL):
    """The extension module, attached to the loaded library; missing, it is an error like a missing library."""
    global _native
    if _native is None:
        try:
            from . import _native as module
        except ImportError as e:
            raise RuntimeError("crusaderbackend_b200._native has not been built (python -m crusaderbackend_b200.build)") from e
        module.attach(lib._handle, CrusaderError)
        _native = module
    return _native


class Context:
    """One cb_ctx on one GPU. `stream=None` binds torch's current stream on that device."""

    def __init__(self, device: int = 0, math: str = "tf32", sync: bool = False, stream: torch.cuda.Stream | None = None):
        self.lib = _lib.load()
        self._native = _load_native(self.lib)
        if not torch.cuda.is_available():
            raise RuntimeError("crusader_b200 needs a CUDA device; there is no CPU path")
        self.device = device
        torch.cuda.set_device(device)
        st = stream if stream is not None else torch.cuda.current_stream(device)
        self._stream = st
        h = C.c_void_p()
        rc = self.lib.cb_create(C.byref(h), device, C.c_void_p(st.cuda_stream))
        if rc != 0:
            raise CrusaderError(rc, "cb_create failed")
        self.h = h
        self._hv = h.value  # what the native calls take
        self.set_math(math)
        self.set_sync(sync)

    # ---- plumbing
    def _check(self, rc: int) -> None:
        if rc != 0:
            raise CrusaderError(rc, self.lib.cb_last_error(self.h).decode())

    def close(self) -> None:
        if getattr(self, "h", None):
            self.lib.cb_destroy(self.h)
            self.h = None
            self._hv = 0

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def set_math(self, math: str) -> None:
        self._check(self.lib.cb_set_math(self.h, MATH_MODES[math]))
        self.math = math

    def set_sync(self, on: bool) -> None:
        self._check(self.lib.cb_set_sync(self.h, int(on)))

    def set_deterministic(self, on: bool) -> None:
        self._check(self.lib.cb_set_deterministic(self.h, int(on)))

    def synchronize(self) -> None:
        self._check(self.lib.cb_synchronize(self.h))

    @property
    def launches(self) -> int:
        return int(self.lib.cb_launch_count(self.h))

    @property
    def last_kernel(self) -> str:
        return self.lib.cb_last_kernel(self.h).decode()

    def measure_umma_peak(self, n: int = 256, p_mn: bool = False, q_mn: bool = False, iters: int = 20000) -> float:
        """TFLOP/s of a resident-operand tcgen05.mma loop (M=128, N=n, K=8, TF32) on every SM."""
        out = C.c_float()
        self._check(self.lib.cb_measure_umma_peak(self.h, n, int(p_mn), int(q_mn), iters, C.byref(out)))
        return float(out.value)

    # ---- GEMM (raw)
    def gemm(self, A: torch.Tensor, B: torch.Tensor, C_: torch.Tensor, transA: bool = False, transB: bool = False,
             accumulate: bool = False) -> torch.Tensor:
        """C = op(A) @ op(B) (+ C). 2-D row-major operands, or 3-D with a leading batch dimension
        (a 2-D A or B is shared by every batch, as in seblas::sgemm)."""
        return self._native.gemm(self._hv, A, B, C_, transA, transB, accumulate)

    # ---- seblas-named GEMMs
    def sgemm(self, A, B, Cout):
        """seblas::sgemm: C[b] = A @ B[b] (seblas/operations/cuGEMM.cu:1649)."""
        return self._native.gemm(self._hv, A, B, Cout, False, False, False)

    def sgemmTN(self, A, B, Cout):
        """seblas::sgemmTN: C[b] = A^T @ B[b], A stored K x M (seblas/operations/cuGEMM.cu:1667)."""
        return self._native.gemm(self._hv, A, B, Cout, True, False, False)

    def sgemmNT(self, A, B, Cout):
        """seblas::sgemmNT: C = A @ B^T, B stored N x K (seblas/operations/cuGEMM.cu:1685)."""
        return self._native.gemm(self._hv, A, B, Cout, False, True, False)

    def sgemmNTA(self, A, B, Cout):
        """seblas::sgemmNTA: C += sum over n of A[n] @ B[n]^T, A n x M x K, B n x N x K, C M x N
        (seblas/operations/cuGEMM.cu:1701); the batch is folded into the contraction, one launch."""
        return self._native.gemm_nta(self._hv, A, B, Cout)

    # ---- convolution: arguments in the order of seblas::conv / convDerive / convError
    def conv(self, A, B, Cout, strideH=1, strideW=1, padH=0, padW=0, biases=None, relu=False):
        """seblas::conv(A=filters OC x IC x FH x FW, B=input N x IC x IH x IW, C=output), seblas/operations/cuConv.cu:757."""
        return self._native.conv(self._hv, A, B, Cout, strideH, strideW, padH, padW, biases, relu)

    def convDerive(self, A, B, Cout, strideH=1, strideW=1, padH=0, padW=0):
        """seblas::convDerive(A=filters, B=dY, C=dX), seblas/operations/cuConv.cu:774."""
        return self._native.conv_dgrad(self._hv, A, B, Cout, strideH, strideW, padH, padW)

    def convError(self, A, B, Cout, strideH=1, strideW=1, padH=0, padW=0, accumulate=True):
        """seblas::convError(A=dY, B=input, C=filter gradient, accumulated), seblas/operations/cuConv.cu:793.
        Returns A, as the reference does."""
        return self._native.conv_wgrad(self._hv, A, B, Cout, strideH, strideW, padH, padW, accumulate)

    def convBias(self, Y, biases):
        return self._native.conv_bias(self._hv, Y, biases)

    def convBiasGrad(self, dY, db, accumulate=False):
        return self._native.conv_bias_grad(self._hv, dY, db, accumulate)

    # ---- linear: seblas::linear / linearXGrad / linearParamGrad (seblas/operations/cuLinear.cu:1052-1115)
    def linear(self, X, W, B, Y):
        return self._native.linear(self._hv, X, W, B, Y)

    def linearXGrad(self, dY, W, dX):
        return self._native.linear_xgrad(self._hv, dY, W, dX)

    def linearParamGrad(self, dY, X, dW, dB):
        return self._native.linear_paramgrad(self._hv, dY, X, dW, dB)

    # ---- neighbours
    def batchNorm(self, X, beta, gamma, mean, var, Y, xHat):
        return self._native.bn_fwd(self._hv, X, beta, gamma, mean, var, Y, xHat)

    def batchNormGrad(self, dY, gamma, X, dX):
        return self._native.bn_bwd(self._hv, dY, gamma, X, dX)

    def batchNormParamGrads(self, dY, xHat, dGamma, dBeta):
        return self._native.bn_paramgrad(self._hv, dY, xHat, dGamma, dBeta)

    def batchNormGradFused(self, dY, gamma, X, dX, dGamma, dBeta, relu_out=None):
        return self._native.bn_bwd_fused(self._hv, dY, gamma, X, dX, dGamma, dBeta, relu_out)

    def batchNormRelu(self, X, beta, gamma, Y):
        return self._native.bn_fwd_relu(self._hv, X, beta, gamma, Y)

    def addRelu(self, A, B, Out):
        return self._native.add_relu(self._hv, A, B, Out)

    def reluGrad2(self, Y, dY, dA, dB=None):
        return self._native.relu_grad2(self._hv, Y, dY, dA, dB)

    def relu(self, X, Y):
        return self._native.relu(self._hv, X, Y)

    def reluGradFast(self, X, dY, dX):
        return self._native.relu_grad(self._hv, X, dY, dX)

    def tensor_op(self, op: int, A, B=None, scalar: float = 0.0):
        return self._native.tensor_op(self._hv, op, A, B, scalar)

    def grad_handover(self, dA, dAReserve):
        return self._native.grad_handover(self._hv, dA, dAReserve)

    def avgPool(self, X, Y, rangeH=2, rangeW=2):
        return self._native.avgpool(self._hv, X, Y, rangeH, rangeW)

    def avgPoolBack(self, dX, dY, rangeH=2, rangeW=2):
        return self._native.avgpool_back(self._hv, dX, dY, rangeH, rangeW)

    def globalAvgPool(self, X, Y):
        return self._native.global_avgpool(self._hv, X, Y)

    def globalAvgPoolBack(self, dX, dY):
        return self._native.global_avgpool_back(self._hv, dX, dY)

    def softmax(self, A, out, step=None):
        return self._native.softmax(self._hv, A, out, step or 0)

    def crossEntropy(self, Y, labels, dY=None, loss=None):
        return self._native.cross_entropy(self._hv, Y, labels, dY, loss)

    def momentumApply(self, X, Xgrad, V, lr, beta, l2=0.0, is_weight=False):
        return self._native.momentum(self._hv, X, Xgrad, V, lr, beta, l2, is_weight)

    def momentumApplyMulti(self, params, grads, moms, is_weight, lr, beta, l2):
        n = len(params)
        arr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
        sizes = (C.c_longlong * n)(*[t.numel() for t in params])
        flags = (C.c_ubyte * n)(*[1 if f else 0 for f in is_weight])
        self._check(self.lib.cb_momentum_multi(self.h, n, arr(params), arr(grads), arr(moms), sizes, flags, lr, beta, l2))
