"""`QuantizedLinear` and `quantized_linear`: the operator API of the W4A16 path.

Drop-in for the reference's `dandan_ops/quantized_linear.py`: same constructor and
factories, buffers (`packed_weight` int32, `scales` float32, `zeros` int32, `bias`),
versioned `extra_state`, load-time validation, dtype pinning, `execution_info` keys and
error messages.  Behind it sits one engine instead of four kernels plus a CPU route:

  * every CUDA FP16 call runs the native library (weight-streaming kernel for small
    batches, tensor-memory GEMM for large ones); the regime is chosen by M, not by a
    backend string or an offline route table;
  * the backend names of the reference are still accepted: "auto", "cuda",
    "tensorcore" and "naive" mean "the engine", "gemv" and "small" keep their M==1 /
    M<=8 argument checks;
  * there is no CPU, BF16, FP32 or training path: what the reference would route to
    its CPU "reference" implementation raises ValueError here, with the reference's own
    wording.

The module keeps the reference-layout tensors (they are the checkpoint format) and a
derived device-native image of them that the kernels read.  The image is rebuilt when
the tensors are replaced or modified in place (load_state_dict, .to()).
"""
import weakref

import torch

from . import _native
from . import ops as _ops_module
from .quantization import (CUDA_ONLY, check_weight, native_quantizer, pack_int4, quantize_int4,
                           read_quantizer_flags, validate_int4_state)

BACKENDS = ("auto", "cuda", "gemv", "small", "tensorcore", "naive", "reference")
FORMAT_VERSION = 2


def _check_bias(bias, rows, device):
    ok = bias is None or (isinstance(bias, torch.Tensor) and bias.ndim == 1 and bias.numel() == rows
                          and bias.device == device and bias.is_floating_point())
    if not ok:
        raise ValueError("bias must be a floating tensor [N] on the input device")


def _resolve(x, scales, group_size, backend):
    """Backend string -> (implementation, reason).  Mirrors the argument checks of
    dandan_ops/quantized_linear.py:17-53; raises where the reference would leave the GPU."""
    if backend not in BACKENDS:
        raise ValueError(f"backend must be one of {BACKENDS}")
    training = torch.is_grad_enabled() and (x.requires_grad or scales.requires_grad)
    if backend == "reference":
        raise ValueError("backend 'reference' does not exist here: this package " + CUDA_ONLY)
    if not (x.is_cuda and x.dtype == torch.float16 and group_size == 64
                                      and not training):
        raise ValueError(CUDA_ONLY)
    if backend == "gemv" and x.shape[0] != 1:
        raise ValueError("gemv requires M=1")
    if backend == "small" and x.shape[0] > 8:
        raise ValueError("small requires M<=8")
    _native.load()
    return None


class _Source:
    """The tensors that something was derived from, held weakly.  They are recognised by themselves: an address, a version and an
    id come back with other tensors.  A copy or a pickle of this knows none."""

    __slots__ = ("refs",)

    def __init__(self, *tensors):
        self.refs = tuple(map(weakref.ref, tensors)) or (lambda: None,) * 3

    def __reduce__(self):
        return _Source, ()


# ------------------------------------------------------------------------------------------
# Native images for callers that hold only reference-layout tensors (the functional form
# and the torch.ops entry points).  Keyed by tensor identity and version counter; entries
# die with their packed weights.
# ------------------------------------------------------------------------------------------
_images = {}


def _state_key(packed, scales, zeros):
    return (packed.data_ptr(), scales.data_ptr(), zeros.data_ptr(),
            packed._version, scales._version, zeros._version, tuple(packed.shape), tuple(scales.shape))


def _image_for(packed, scales, zeros, in_features):
    ident = id(packed)
    entry = _images.get(ident)
    key = _state_key(packed, scales, zeros)
    if entry is not None and entry[0] == key and entry[1]() is packed and entry[2]() is scales and entry[3]() is zeros:
        return entry[4]
    image = _native.repack(packed, scales, zeros, in_features)
    ref = weakref.ref(packed, lambda _r, i=ident: _images.pop(i, None))
    _images[ident] = (key, ref, weakref.ref(scales), weakref.ref(zeros), image)
    return image


def _engine(x, image, rows, in_features, bias16, flags=0):
    """`bias16`: the bias already converted to FP16 (or None); `flags`: layer flags of the C ABI.  The kernels round the product to
    FP16 first and add the FP16 bias afterwards, as the reference's `y + bias.to(y.dtype)` does."""
    if x.stride(1) != 1 or (x.shape[0] > 1 and x.stride(0) < in_features):
        x = x.contiguous()
    if _ops_module.SHIM_LOADED:       # C++ operator library: output, workspace and launch without a ctypes round trip
        return _ops_module.linear_image(x, image, rows, in_features, bias16, 0, flags)
    return _native.linear(x, image, rows, in_features, bias=bias16, flags=flags)


def quantized_linear(x, packed_weight, scales, zeros, *, in_features, group_size=64, bias=None,
                     backend="auto"):
    """y = fp16(x @ W^T) (+ bias) with W = fp16((code - zero) * step), FP32 accumulation
    (dandan_ops/quantized_linear.py:56-81).  CUDA FP16 activations only."""
    validate_int4_state(packed_weight, scales, zeros, in_features, group_size)
    if not isinstance(x, torch.Tensor) or x.ndim != 2 or x.shape[1] != in_features:
        raise ValueError("x must have shape [M, in_features]")
    if x.dtype not in (torch.float16, torch.bfloat16, torch.float32):
        raise TypeError("x must be float16, bfloat16, or float32")
    if x.device != packed_weight.device:
        raise ValueError("x and quantized weight must share a device")
    _check_bias(bias, packed_weight.shape[0], x.device)
    _resolve(x, scales, group_size, backend)
    image = _image_for(packed_weight.contiguous(), scales.contiguous(), zeros.contiguous(), in_features)
    bias16 = None if bias is None else bias.to(torch.float16).contiguous()
    return _engine(x, image, packed_weight.shape[0], in_features, bias16)


class QuantizedLinear(torch.nn.Module):
    """Packed INT4 linear layer (inference only).

    Values are validated when the layer is built or a checkpoint is loaded (that
    synchronizes); `forward` checks metadata only and never reads tensor values on the
    host, so it can be captured into a CUDA graph and replayed.
    """

    def __init__(self, packed_weight, scales, zeros, *, in_features, group_size=64, bias=None,
                 backend="auto", defer_image=False):
        """`defer_image=True` (an addition to the reference's signature) skips the eager build of the
        device-native image: for loaders that attach a prebuilt one (`checkpoint.ImageCache.load_layer`)."""
        super().__init__()
        if backend not in BACKENDS:
            raise ValueError("invalid quantized backend")
        validate_int4_state(packed_weight, scales, zeros, in_features, group_size, values=True)
        self._set_state(packed_weight, scales, zeros, in_features, group_size, bias, backend)
        if self.packed_weight.is_cuda and group_size == 64 and not defer_image:
            self._native_image()

    def _set_state(self, packed_weight, scales, zeros, in_features, group_size, bias, backend):
        """Attributes and buffers of a layer whose quantized state is known to be valid."""
        _check_bias(bias, packed_weight.shape[0], packed_weight.device)
        # plain attributes go straight into the instance (Module.__setattr__ looks for parameters and submodules)
        self.__dict__.update(in_features=in_features, out_features=packed_weight.shape[0], group_size=group_size,
                             backend=backend, _image=None, _image_key=None, _image_flags=0, _bias16=None,
                             _bias16_key=None, _checked_key=None, _checked_device=None, training=False)
        self.register_buffer("packed_weight", packed_weight.detach().contiguous())
        self.register_buffer("scales", scales.detach().contiguous())
        self.register_buffer("zeros", zeros.detach().contiguous())
        self.register_buffer("bias", None if bias is None else bias.detach().clone().contiguous())

    # -- construction ----------------------------------------------------------------------
    @classmethod
    def from_float(cls, weight, bias=None, *, bits=4, group_size=64, backend="auto"):
        """Quantize a floating-point [N, K] weight (dandan_ops/quantized_linear.py:158-165)."""
        if not isinstance(bits, int) or isinstance(bits, bool) or bits != 4:
            raise ValueError("only bits=4 is supported")
        check_weight(weight)
        if (native_quantizer(weight, group_size) and backend in BACKENDS and cls.__init__ is QuantizedLinear.__init__):
            # One pass gives the state and the image of it.  Its steps are positive normal FP32 numbers and its zero
            # points 0..15 by construction, so nothing is read back to check them.
            with torch.no_grad():
                source = weight.detach().contiguous()
                if (_ops_module.SHIM_LOADED and type(source) is torch.Tensor
                        and not torch._C._functorch.is_functorch_wrapped_tensor(source)):
                    packed, steps, zero_points, image, flags = _ops_module.quantize_image(source)
                else:
                    _, packed, steps, zero_points, image, flags = _native.quantize(source)
                layer = cls.__new__(cls)                      # (built while the kernel runs)
                torch.nn.Module.__init__(layer)
                layer._set_state(packed, steps, zero_points, weight.shape[1], group_size, bias, backend)
                key, source = layer._state_key(), _Source(*layer._state())
                layer._set_image(image, key, source, read_quantizer_flags(flags))
            return layer
        with torch.no_grad():
            codes, steps, zero_points = quantize_int4(weight, group_size)
        return cls(pack_int4(codes), steps, zero_points, in_features=weight.shape[1],
                   group_size=group_size, bias=bias, backend=backend)

    @classmethod
    def from_state_dict(cls, state, *, backend="auto"):
        meta = state.get("_extra_state")
        if not isinstance(meta, dict) or meta.get("format_version") != FORMAT_VERSION:
            raise ValueError("missing or unsupported INT4 format_version")
        shape = meta.get("original_shape")
        if not isinstance(shape, (tuple, list)) or len(shape) != 2:
            raise ValueError("invalid original_shape metadata")
        layer = cls(state["packed_weight"], state["scales"], state["zeros"], in_features=shape[1],
                    group_size=meta["group_size"], bias=state.get("bias"), backend=backend)
        layer.load_state_dict(state)
        return layer

    # -- checkpoint format -----------------------------------------------------------------
    def get_extra_state(self):
        return {"format_version": FORMAT_VERSION, "bits": 4, "scheme": "affine_unsigned",
                "packing": "int32_low_nibble_first",
                "original_shape": [self.out_features, self.in_features],
                "group_size": self.group_size, "fp16_weight_rounding": "fp16_before_multiply"}

    def set_extra_state(self, state):
        mine = self.get_extra_state()
        if not isinstance(state, dict) or any(state.get(k) != v for k, v in mine.items()):
            raise ValueError("incompatible INT4 checkpoint metadata/version/shape/group_size")

    def _load_from_state_dict(self, state_dict, prefix, local_metadata, strict, missing_keys,
                              unexpected_keys, error_msgs):
        # Validate everything before anything is copied: a bad checkpoint must leave the
        # layer untouched (dandan_ops/quantized_linear.py:115-130).
        names = [prefix + n for n in ("packed_weight", "scales", "zeros")]
        try:
            self.set_extra_state(state_dict.get(prefix + "_extra_state"))
            if all(n in state_dict for n in names):
                validate_int4_state(state_dict[names[0]], state_dict[names[1]], state_dict[names[2]],
                                    self.in_features, self.group_size, values=True)
                if state_dict[names[0]].shape[0] != self.out_features:
                    raise ValueError("incompatible output dimension")
            bias = state_dict.get(prefix + "bias")
            if bias is not None:
                _check_bias(bias, self.out_features, state_dict[names[0]].device)
        except (ValueError, TypeError, KeyError) as exc:
            error_msgs.append(f"{prefix}invalid INT4 state: {exc}")
            return
        super()._load_from_state_dict(state_dict, prefix, local_metadata, strict, missing_keys,
                                      unexpected_keys, error_msgs)

    def _apply(self, fn, recurse=True):
        # .half()/.bfloat16()/.to(dtype) must not touch the quantized state: keep the
        # original tensors and only follow the device (dandan_ops/quantized_linear.py:148-156).
        words, steps, zero_points = self.packed_weight, self.scales, self.zeros
        super()._apply(fn, recurse=recurse)
        device = self.packed_weight.device
        self.packed_weight = words.to(device=device, dtype=torch.int32)
        self.scales = steps.to(device=device, dtype=torch.float32)
        self.zeros = zero_points.to(device=device, dtype=torch.int32)
        return self

    # -- native image ----------------------------------------------------------------------
    def _state(self):
        # (the buffers where Module keeps them: its attribute lookup takes longer than the rest of a key)
        buffers = self._buffers
        try:
            return buffers["packed_weight"], buffers["scales"], buffers["zeros"]
        except KeyError:                                     # turned into parameters or plain attributes
            return self.packed_weight, self.scales, self.zeros

    def _state_key(self):
        packed, scales, zeros = self._state()
        return (packed.data_ptr(), scales.data_ptr(), zeros.data_ptr(), packed._version, scales._version, zeros._version)

    _slice_flag = 0
    _image_source = _bias16_source = _Source()

    def serve_as_column_slice(self):
        """This layer is one rank's slice of a column-sharded layer: up to 16 rows of x every call runs the kernels that
        carry the all-gather, so that the slice has the same bits in every form of the gather (FLAG_COLUMN_SLICE)."""
        self._slice_flag = _native.FLAG_COLUMN_SLICE
        self._image_flags |= self._slice_flag

    def _set_image(self, image, key, source, found):
        """Adopt an image of the state with this key that is complete in memory (its stream has been synchronized); `found`: its
        QUANT_* bits."""
        self._adopt(image, key, source, _native.step_flags(found))

    def _adopt(self, image, key, source, flags):
        # (in one step, and past Module's attribute hook, which takes about a microsecond per name)
        self.__dict__.update(_image=image, _image_key=key, _image_source=source, _image_flags=flags | self._slice_flag, _checked_key=None)

    def _native_image(self):
        key = self._state_key()
        packed, scales, zeros = self._state()
        of_packed, of_scales, of_zeros = self._image_source.refs
        if self._image is None or self._image_key != key or of_packed() is not packed or of_scales() is not scales or of_zeros() is not zeros:
            image = _native.repack(packed, scales, zeros, self.in_features)
            self._adopt(image, key, _Source(packed, scales, zeros), self._layer_flags(image))
        return self._image

    def _layer_flags(self, image=None):
        """Flags of the C ABI for an image of this layer (that at hand).  FLAG_FP16_STEPS when every step is exactly representable in
        FP16 (checkpoints with FP16 scales): the decode kernels then use the FP16-only dequantization, which
        is bit-identical for such steps; FLAG_PLAIN_STEPS when none is factored; FLAG_OVERLAP_LAUNCH unless switched off
        (B2_W4A16_OVERLAP=0).  Reads the image's steps once (a host sync), only when an image is (re)built -
        never on the per-token path - and not while a stream is being captured."""
        if not self.scales.is_cuda or torch.cuda.is_current_stream_capturing():
            return 0
        # The read synchronizes the stream, so the image is complete in memory from here on: the
        # decode kernel may start under the tail of whatever kernel precedes it (FLAG_OVERLAP_LAUNCH).
        return _native.step_flags(_native.image_flags(self._image if image is None else image, self.out_features, self.in_features))

    def attach_native_image(self, image, factored=True):
        """Use a prebuilt device image of THIS layer's state (e.g. from `checkpoint.ImageCache`)
        instead of repacking.  The image is dropped again if the state tensors change.  `factored=False` asserts that
        none of its steps is factored (FLAG_PLAIN_STEPS)."""
        if image.dtype != torch.uint8 or image.device != self.packed_weight.device or \
                image.numel() != _native.native_bytes(self.out_features, self.in_features):
            raise ValueError("not a native image of this layer")
        flags = 0
        if self.scales.is_cuda and not torch.cuda.is_current_stream_capturing():
            fp16 = bool((self.scales.half().float() == self.scales).all())             # (synchronizes, as _layer_flags)
            flags = _native.step_flags((0 if fp16 else _native.QUANT_STEP_NOT_FP16) | (_native.QUANT_FACTORED if factored else 0))
        self._adopt(image, self._state_key(), _Source(*self._state()), flags)

    def _bias_fp16(self):
        """FP16 copy of the bias for the fused epilogue (derived, rebuilt when the bias changes)."""
        bias = self._bias()
        if bias is None:
            return None
        key = (bias.data_ptr(), bias._version, bias.dtype)
        if self._bias16 is None or self._bias16_key != key or self._bias16_source.refs[0]() is not bias:
            self.__dict__.update(_bias16=bias.detach().to(torch.float16).contiguous(), _bias16_key=key, _bias16_source=_Source(bias))
        return self._bias16

    # -- introspection ---------------------------------------------------------------------
    def execution_info(self, x):
        """What `forward(x)` would run, without running it (same keys as the reference;
        `kernel_plan` is an addition)."""
        try:
            _resolve(x, self.scales, self.group_size, self.backend)
        except ValueError as exc:
            return {"requested_backend": self.backend, "implementation": "unavailable",
                    "fallback_reason": str(exc), "reason": str(exc), "input_copies": [],
                    "format_version": FORMAT_VERSION, "activation_dtype": str(x.dtype),
                    "group_size": self.group_size, "kernel_plan": None}
        plan = _native.plan(x.shape[0], self.out_features, self.in_features, self._slice_flag)
        return {"requested_backend": self.backend, "implementation": plan["route"],
                "fallback_reason": None, "reason": "selected packed inference backend",
                "input_copies": [i for i, t in enumerate((x, self.packed_weight, self.scales, self.zeros))
                                 if not t.is_contiguous()],
                "format_version": FORMAT_VERSION, "activation_dtype": str(x.dtype),
                "group_size": self.group_size, "kernel_plan": plan}

    @property
    def storage_bytes(self):
        """Bytes of the checkpoint-format state, as the reference counts them."""
        return sum(t.numel() * t.element_size() for t in (self.packed_weight, self.scales, self.zeros))

    @property
    def native_bytes(self):
        """Bytes of the device image the kernels stream (0.5703 B/weight for full tiles)."""
        return _native.native_bytes(self.out_features, self.in_features)

    def dequantize(self):
        """FP32 [N, K] weights, bit-identical to the reference's dequantize_int4."""
        if not self.packed_weight.is_cuda or self.group_size != 64:
            raise ValueError("dequantize " + CUDA_ONLY.replace(" FP16", ""))
        return _native.dequantize(self._native_image(), self.out_features, self.in_features)

    def _bias(self):
        buffers = self._buffers                              # (as _state: a lookup through Module takes half a microsecond)
        return buffers["bias"] if "bias" in buffers else self.bias

    def _forward_key(self, packed, scales, zeros, bias):
        return (packed.data_ptr(), scales.data_ptr(), zeros.data_ptr(),
                packed._version, scales._version, zeros._version,
                self.in_features, self.group_size, self.backend,
                None if bias is None else (bias.data_ptr(), bias._version, bias.dtype))

    def forward(self, x):
        # Per-token fast path: the metadata checks below depend only on the layer's state, so they
        # are repeated only when a state tensor was replaced or written (the tensor itself, data pointer,
        # version counter), an attribute was reassigned, or x is not the plain CUDA FP16 case.
        packed, scales, zeros = self._state()
        bias = self._bias()
        key = self._forward_key(packed, scales, zeros, bias)
        of_packed, of_scales, of_zeros = self._image_source.refs       # (a new image takes the checked key back)
        if (key == self._checked_key and of_packed() is packed and of_scales() is scales and of_zeros() is zeros
                and (bias is None or (self._bias16_key == key[-1] and self._bias16_source.refs[0]() is bias))
                and type(x) is torch.Tensor and x.dtype is torch.float16 and x.ndim == 2
                and x.shape[1] == self.in_features and x.device == self._checked_device
                and not (x.requires_grad and torch.is_grad_enabled())):
            return _engine(x, self._image, self.out_features, self.in_features, None if bias is None else self._bias16, self._image_flags)
        y = self._forward_checked(x)
        if self.backend in ("auto", "cuda", "tensorcore", "naive") and not self.scales.requires_grad \
                and self._image is not None:
            packed, scales, zeros = self._state()
            self.__dict__.update(_checked_key=self._forward_key(packed, scales, zeros, self._bias()), _checked_device=packed.device)
        return y

    def check_input(self, x):
        """Metadata checks of the raw-kernel entry points (`forward_into`, the sharded layer's fused call):
        CUDA FP16 `[M, in_features]`; returns x with unit inner stride."""
        if type(x) is not torch.Tensor or x.dtype is not torch.float16 or x.ndim != 2 or x.shape[1] != self.in_features:
            raise ValueError("x must be a CUDA FP16 tensor [M, in_features]")
        _resolve(x, self.scales, self.group_size, self.backend)
        if x.stride(1) != 1 or (x.shape[0] > 1 and x.stride(0) < self.in_features):
            x = x.contiguous()
        return x

    def forward_into(self, x, out):
        """`forward(x)` written into `out`, an FP16 `[M, N]` CUDA tensor or a column slice of a wider one
        (unit inner stride; the row stride is passed to the kernel).  Used by the column-sharded layer,
        whose slice of the gathered output lives in memory shared with the other ranks."""
        if (out.dtype != torch.float16 or out.ndim != 2 or tuple(out.shape) != (x.shape[0], self.out_features)
                or out.stride(1) != 1 or out.device != x.device):
            raise ValueError("out must be an FP16 [M, N] tensor with unit inner stride on the input device")
        x = self.check_input(x)
        image = self._native_image()
        return _native.linear(x, image, self.out_features, self.in_features, out=out, bias=self._bias_fp16(),
                              flags=self._image_flags)

    def _forward_checked(self, x):
        validate_int4_state(self.packed_weight, self.scales, self.zeros, self.in_features, self.group_size)
        if not isinstance(x, torch.Tensor) or x.ndim != 2 or x.shape[1] != self.in_features:
            raise ValueError("x must have shape [M, in_features]")
        if x.dtype not in (torch.float16, torch.bfloat16, torch.float32):
            raise TypeError("x must be float16, bfloat16, or float32")
        if x.device != self.packed_weight.device:
            raise ValueError("x and quantized weight must share a device")
        _check_bias(self.bias, self.out_features, x.device)
        _resolve(x, self.scales, self.group_size, self.backend)
        image = self._native_image()
        return _engine(x, image, self.out_features, self.in_features, self._bias_fp16(), self._image_flags)
