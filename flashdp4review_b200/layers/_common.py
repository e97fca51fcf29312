"""Shared pieces of the DP layer backward passes."""
import weakref

import torch

from .. import _lib, runtime
from ..core import ops
from ..core.ops import NoiseSpec, noise_std
from ..distributed import direct_reducer


class DPLayerMixin:
    """Hyper-parameters and noise bookkeeping common to the DP layers."""

    def _init_dp(self, C, clamp_value, noise_multiplier, n_tensors=2):
        self.dp = True
        self.C = C
        self.clamp_value = clamp_value
        self.noise_multiplier = noise_multiplier
        self._dp_param_ids = [runtime.next_param_id() for _ in range(n_tensors)]
        self._dp_step = 0

    def _next_step(self):
        # (past nn.Module's __setattr__, which takes as long as the rest of a backward's bookkeeping)
        d = self.__dict__
        step = d["_dp_step"] = d["_dp_step"] + 1
        return runtime.noise_step(step)


def reshape_to_3d(input, grad_output):
    """(B,T,.) views of the saved input and the upstream gradient: 2-D gets T=1, >3-D folds the
    middle axes into T (flashdp/layers/linear.py:51-58)."""
    if input.dim() == 2:
        return input.unsqueeze(1), grad_output.unsqueeze(1)
    if input.dim() > 3:
        B = input.shape[0]
        return input.reshape(B, -1, input.shape[-1]), grad_output.reshape(B, -1, grad_output.shape[-1])
    return input, grad_output


def dp_scalars(local_batch, noise_multiplier, param_id, step, param_id2=0):
    """(batch_divisor, NoiseSpec) for one backward call under the current run layout."""
    rank, world = runtime.data_parallel()
    micro_index, micro_steps = runtime.accumulation()
    global_batch = local_batch * world * micro_steps
    # under gradient accumulation only the last micro-step carries the (single) noise draw
    std = noise_std(noise_multiplier, global_batch) if micro_index == micro_steps - 1 else 0.0
    return global_batch, NoiseSpec(std=std, seed=runtime.get_seed(),
                                   param_id=param_id, param_id2=param_id2, step=step, rank=rank, world=world,
                                   step_device=runtime.device_noise_counter() if std != 0.0 else None)


def direct_grad_target(param):
    """The bucket slice a DP weight gradient may be written into directly, or None.

    A DPGradReducer built with grad_as_bucket_view=True offers the slice once per accumulation
    cycle (the first gradient of the cycle overwrites it: no zero fill, no accumulate pass by
    autograd); later gradients of the same cycle go the ordinary way and are added by autograd.
    """
    reducer = direct_reducer(param)
    return reducer.claim_direct(param) if reducer is not None else None


def direct_grad_done(param):
    """Tell the reducer that the gradient written into the claimed slice is complete (queued on
    the current stream), as autograd's post-accumulate hook would have."""
    direct_reducer(param).direct_written(param)


def autocast_dtype(*tensors):
    """The CUDA autocast dtype if autocast is on and the tensors live on a GPU, else None.

    Under autocast the DP layers behave like their plain twins (nn.Linear, Conv1D): operands are
    cast to the autocast dtype in forward, the output comes out in it, and the cast input is what
    backward sees -- so the upstream gradient is 16-bit and the tensor-core kernels run.  (In the
    reference the Conv1D forward adds an fp32 bias to the bf16 product, the output and hence the
    whole backward become fp32 -- flashdp/layers/transformers_conv1d.py:40-43.)
    """
    if torch.is_autocast_enabled("cuda") and all(t is None or t.is_cuda for t in tensors):
        return torch.get_autocast_dtype("cuda")
    return None


# ---- the native autograd nodes (csrc/fdp_host.cpp) and what they ask Python for ------------------------------------
_CODES = {code: dtype for dtype, code in ops._DT.items()}
_native = None


def native_nodes(input):
    """The call layer with the layers' autograd nodes, or None where the Function classes take the call: tensors that
    are not on a GPU, and torch.jit.trace, which records a Function but would take a node's output for a constant."""
    global _native
    if not input.is_cuda or torch._C._get_tracing_state() is not None:
        return None
    if _native is None:
        host = _lib.host()
        host.bind_layers({"product": _product, "linear": _linear_call, "layernorm": _layernorm_call,
                          "direct_done": direct_grad_done, "check": _lib.check, "dtype": lambda t: ops._dt(t.dtype)})
        _native = host
    return _native


class _NodeState:
    """What a native node holds of its layer.  Not the layer itself: Python's collector does not see through such a node,
    and a layer that keeps an output of its own (a hook that captures activations) would be kept alive by it, with its
    parameters and the graph.  The layer is asked as long as it lives; once it is gone, what it was at its last
    forward holds, and all of its nodes count their steps on from there."""
    __slots__ = ("layer", "C", "clamp_value", "noise_multiplier", "norm_algo", "_dp_param_ids", "_dp_step")

    def __init__(self, layer):
        self.layer = weakref.ref(layer)

    def _next_step(self):
        self._dp_step += 1
        return runtime.noise_step(self._dp_step)

    def follow(self, layer):
        self.C, self.clamp_value, self.noise_multiplier = layer.C, layer.clamp_value, layer.noise_multiplier
        self._dp_param_ids, self._dp_step = layer._dp_param_ids, layer._dp_step
        self.norm_algo = getattr(layer, "norm_algo", "auto")


_states = weakref.WeakKeyDictionary()      # one state a living layer


def node_state(layer):
    """The state that the nodes of this forward hold."""
    state = _states.get(layer)
    if state is None:
        state = _states.setdefault(layer, _NodeState(layer))
    state.follow(layer)
    return state


def _step_of(state):
    """The layer, or its state if it is gone, and the step of this backward."""
    layer = state.layer()
    if layer is None:
        return state, state._next_step()
    step = layer._next_step()
    state._dp_step = layer._dp_step
    return layer, step


def _product(code, rows, K, N):
    return ops.library_product_ok(_CODES[code], rows, K, N)


def _linear_call(state, weight, B, code, rows, K, N, need_dx, need_dw, need_db):
    """One backward of a Linear / Conv1D layer: whether the input gradient is the library's and, if the call is for
    anything of the library's, the parameters of the weight's and of the bias's gradient, the flags of the call, and the
    bucket slice the weight gradient goes to.  `code` is -1 for a dtype that the kernels do not know."""
    layer, step = _step_of(state)
    native_dx = need_dx and code >= 0 and ops.library_product_ok(_CODES[code], rows, K, N)
    if not (native_dx or need_dw or need_db):
        return (False,)                  # (an empty batch of a frozen layer, for one, has no noise to form)
    w_id, b_id = layer._dp_param_ids
    div, noise = dp_scalars(B, layer.noise_multiplier, w_id, step)
    p = ops._params(layer.C, layer.clamp_value, div, noise)
    bias = p[:5] + (int(b_id) & 0xFFFFFFFF,) + p[6:]
    return native_dx, p, bias, ops.backward_algo(code, layer.norm_algo), direct_grad_target(weight) if need_dw else None


def _layernorm_call(state, B):
    layer, step = _step_of(state)
    g_id, b_id = layer._dp_param_ids
    div, noise = dp_scalars(B, layer.noise_multiplier, g_id, step, param_id2=b_id)
    return ops._params(layer.C, layer.clamp_value, div, noise)
