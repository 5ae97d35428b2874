"""Newton-Schulz engine: the object the optimizer routes every matrix through.

Drop-in for the reference's ``CutlassNSInt8`` (src/i8muon/_cutlass.py:15-49):
same constructor arguments, the same four entry points ``_regular_prec``,
``_gram_prec``, ``_regular_i8`` and ``_regular_bq`` with the call convention
``fn(x, coeffs=None, eps=1e-7, deterministic=True, precision=...) -> Tensor``
(same shape and dtype as ``x``; leading dimensions fold into the batch), and the
same ``router``.  Each entry point is one call into the sm_100a library
(``i8m_ns_run``), which sequences the fused kernels on the current stream.

Differences that a caller can observe:
  * only compute capability 10.x devices are accepted;
  * ``deterministic=False`` selects one-pass statistics with atomics on every route (the reference
    only has that flavour for global INT8); the default is the two-pass reduction in a fixed order;
  * the result is a fresh tensor, not a view into the call's workspace;
  * with ``deterministic=True`` a matrix's result has the same bits alone and in any batch, in every precision;
  * ``tiles`` selects, per product of the global-INT8 route (``aat``, ``square``, ``update``), between this
    library's kernels for whole-K products: the reference's tile id 4 (its TMA tile) maps to the
    persistent kernel with 128 x 256 units (also the default), ids 0-3 (its cp.async tiles) to the
    one-CTA-per-tile kernel;
    ``autotune`` times the library's kernel variants (``tuning.py``).
"""
from __future__ import annotations

import contextlib
import ctypes
import math
import os

import torch

from . import native
from .coefficients import DEFAULT_COEFFICIENTS
from .routing import matrix_spec, normalize_precision, select_route
from .tuning import KernelFactory

_COMPUTE_CODES = {"float32": native.F32, "float16": native.F16, "bfloat16": native.BF16}
_STATUS_WORDS = {}


def status_word(device: torch.device) -> torch.Tensor:
    """One zeroed int32 per device that kernels write an error code to when a
    bounded device-side wait gives up."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    word = _STATUS_WORDS.get(index)
    if word is None:
        # setdefault: of two threads that come here together both get the word that stays (its address is kept)
        word = _STATUS_WORDS.setdefault(index, torch.zeros(1, dtype=torch.int32, device=torch.device("cuda", index)))
    return word


def check_status(device=None) -> None:
    """Synchronise and raise if any kernel on ``device`` reported a timed-out wait."""
    devices = list(_STATUS_WORDS) if device is None else [torch.device(device).index or 0]
    for index in devices:
        word = _STATUS_WORDS.get(index)
        if word is None:
            continue
        code = int(word.item())
        if code:
            word.zero_()
            raise native.NativeError(f"device-side wait timed out, status word 0x{code:x}")


_STATUS_HOST = {}


def status_host(index: int) -> torch.Tensor:
    """One int32 in pinned host memory per device, where the status word is copied to at the end of a step."""
    host = _STATUS_HOST.get(index)
    if host is None:
        host = _STATUS_HOST.setdefault(index, torch.zeros(1, dtype=torch.int32).pin_memory())
        _STATUS_VIEWS[index] = ctypes.c_int32.from_address(host.data_ptr())
    return host


_STATUS_VIEWS = {}   # the same words as ctypes integers: reading one is a plain load


def post_status(device) -> None:
    """Queue a copy of the device's status word to pinned host memory on the current stream; nothing
    waits for it.  ``raise_if_reported`` looks at the copy once it has landed."""
    index = torch.device(device).index
    index = torch.cuda.current_device() if index is None else index
    word = _STATUS_WORDS.get(index)
    if word is None or torch.cuda.is_current_stream_capturing():
        return
    host = status_host(index)
    with torch.cuda.device(index):
        host.copy_(word, non_blocking=True)


def raise_if_reported() -> None:
    """Raise if a status word copied to the host has arrived and is not zero (no synchronisation)."""
    for index, view in tuple(_STATUS_VIEWS.items()):
        code = view.value
        if code != 0:
            torch.cuda.synchronize(index)   # copies still in flight land before the words are cleared
            _STATUS_WORDS[index].zero_()
            view.value = 0
            raise native.NativeError(f"device-side wait timed out on cuda:{index}, status word 0x{code:x}; the "
                                     "results of the previous step are incomplete")


# raw handle of the current stream of a device; the public spelling builds a Stream object for every call
raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (
    lambda index: torch.cuda.current_stream(index).cuda_stream)
_current_device = getattr(torch._C, "_cuda_getDevice", None) or torch.cuda.current_device
_NO_SWITCH = contextlib.nullcontext()


def on_device(index: int):
    """Context in which CUDA device ``index`` is current (free when it already is)."""
    return _NO_SWITCH if _current_device() == index else torch.cuda.device(index)


def gram_order() -> str:
    order = os.environ.get("I8MUON_GRAM_RESET", "00100")
    if not order or order[0] != "0" or set(order) - {"0", "1"}:
        raise ValueError("I8MUON_GRAM_RESET must be a binary string starting with 0")
    return order


_COEFFICIENT_ARRAYS = {}
MAX_COEFFICIENT_ARRAYS = 256


def keep(table: dict, limit: int, key, value) -> None:
    """Put ``value`` into a bounded table; the entry that has been there longest makes room."""
    while len(table) >= limit:
        table.pop(next(iter(table)), None)
    table[key] = value


def coefficient_rows(coeffs):
    """The rows as tuples of floats: what a schedule is known by."""
    return tuple([tuple(map(float, row)) for row in coeffs])


def coefficient_array(coeffs):
    """The rows as a C array and their number; the arrays of recent schedules are kept."""
    key = coefficient_rows(coeffs)
    hit = _COEFFICIENT_ARRAYS.get(key)
    if hit is None:
        if not key or any(len(row) != 3 for row in key):
            raise ValueError("Expected a nonempty list of (a, b, c) coefficients")
        flat = [v for row in key for v in row]
        hit = (ctypes.c_double * len(flat))(*flat), len(key)
        keep(_COEFFICIENT_ARRAYS, MAX_COEFFICIENT_ARRAYS, key, hit)
    return hit


class CutlassNSInt8:
    """Native floating-point regular/Gram NS and regular INT8 / INT8-BQ / FP8-BQ NS."""

    def __init__(self, autotune=False, *, tiles=None, fp16_first=True):
        self.fp16_first = fp16_first
        self.autotune = autotune
        self.tiles = dict(tiles or {})
        # kernel selection of calls that neither ``tiles`` nor the tuner decides, in i8m_ns_run's packing
        # (block-quantised GEMM | whole-K GEMM << 8 | its square << 16 | its update << 24); 0: the defaults
        # (environment I8MUON_B200_KERNEL_VARIANTS presets it: an integer, e.g. 0x02020200)
        self.kernel_variants = int(os.environ.get("I8MUON_B200_KERNEL_VARIANTS", "0"), 0)
        if (set(self.tiles) - {"aat", "square", "update"}
                or any(v not in (0, 1, 2, 3, 4) for v in self.tiles.values())):
            raise ValueError("tiles accepts aat/square/update with values 0/1/2/3/4")
        self._routes = {}
        self._specs = {}         # checked geometry and workspace size of the calls seen so far
        self._group_plans = {}   # native plans of the optimizer's shape groups (optimizer.py)
        self._factory = KernelFactory(autotune)

    def __getstate__(self):
        """What a copy or a pickle of the engine carries: its settings and measurements.  The tables below hold
        addresses of this process (status words, coefficient arrays) and are built again where they are needed."""
        return {**self.__dict__, "_routes": {}, "_specs": {}, "_group_plans": {}}

    # ------------------------------------------------------------ routing
    def router(self, M: int, N: int, precision: str, use_gram: bool, gram_aspect_threshold: float):
        key = (M, N, precision, use_gram, gram_aspect_threshold)
        hit = self._routes.get(key)
        if hit is None:
            name, compute = select_route(M, N, precision, use_gram, gram_aspect_threshold)
            hit = self._routes[key] = (getattr(self, name), compute)
        return hit

    # ------------------------------------------------------------- launch
    def _run(self, route, x, coeffs, eps, compute, alignment, spec_precision, fp16_first, out=None,
             deterministic=True, stats=None):
        array, steps = coefficient_array(DEFAULT_COEFFICIENTS if coeffs is None else coeffs)
        shape, device = x.shape, x.device
        spec = (route, shape, x.dtype, device, compute, steps, alignment, spec_precision, bool(fp16_first))
        known = self._specs.get(spec)
        if known is None:
            batch, rows, cols, *_ = matrix_spec(tuple(shape), x.dtype, device, spec_precision, alignment)
            dtype = native.torch_dtype_code(x.dtype)
            with on_device(device.index):
                size = native.ns_workspace_bytes(route, batch, rows, cols, dtype, compute, steps, fp16_first)
            known = batch, rows, cols, dtype, size, status_word(device).data_ptr()
            if len(self._specs) < 1024:
                self._specs[spec] = known
        batch, rows, cols, dtype, size, status = known
        x = x.contiguous()
        order = gram_order().encode() if route == native.ROUTE_GRAM else None
        with on_device(device.index):
            if out is None:
                out = torch.empty_like(x)
            elif (out.shape != x.shape or out.dtype != x.dtype or out.device != x.device
                  or not out.is_contiguous() or out.data_ptr() == x.data_ptr()):
                raise ValueError("out must be a contiguous tensor like x that does not alias it")
            if stats is not None and (stats.dtype != torch.float32 or stats.device != x.device or not stats.is_contiguous()
                                      or stats.numel() * 4 < native.stats_scratch_bytes(batch, rows * cols)):
                raise ValueError("stats must be the FP32 partials that i8m_momentum left for x")

            def launch(variant):
                workspace = torch.empty(size, dtype=torch.uint8, device=device)
                native.call("i8m_ns_run", route, x.data_ptr(), out.data_ptr(), dtype, batch, rows, cols,
                            compute, array, steps, float(eps), int(bool(fp16_first)), int(bool(deterministic)),
                            int(variant), order, stats.data_ptr() if stats is not None else None,
                            workspace.data_ptr(), size, status, raw_stream(device.index))

            variant = self.kernel_variants
            if route in (native.ROUTE_INT8, native.ROUTE_INT8_FACTORED) and self.tiles:
                # explicit tiles take precedence over measurements, as in the reference
                per_op = [0 if self.tiles.get(op, 4) == 4 else 2 for op in ("aat", "square", "update")]
                variant = (per_op[0] << 8) | (per_op[1] << 16) | (per_op[2] << 24)
            elif self._factory.autotune:
                # per operation first (median of three graph replays, >= 2 % to replace the default), then the
                # tuned call as a whole against the all-default call (>= 1 %), as the reference's factory does
                key = (device.index, x.dtype, batch, rows, cols, route, compute, steps, bool(fp16_first))
                tuned = 0
                if route in (native.ROUTE_BQ_INT8, native.ROUTE_BQ_FP8):
                    tuned = self._factory.select("bq_gemm", key, tuple(range(native.variant_count("bq_gemm"))), 0, launch)
                if route != native.ROUTE_BQ_FP8 and not (route == native.ROUTE_FLOAT and compute == native.F32):
                    # routes with whole-K products (the FP16 first row included): bits 8.. select their kernel
                    choice = self._factory.select("wholek_gemm", key, tuple(range(native.variant_count("wholek_gemm"))), 0,
                                                  lambda v: launch(tuned | (v << 8) | (v << 16) | (v << 24)))
                    tuned |= (choice << 8) | (choice << 16) | (choice << 24)
                if tuned and self._factory.select_pipeline("ns_call", key, lambda use: launch(tuned if use else 0)):
                    variant = tuned
            launch(variant)
        # The workspace may be reused by later allocations on this stream only.
        return out.view(shape)

    def call_spec(self, name: str, precision: str):
        """(route, compute code, alignment, precision name of the geometry check, fp16_first) of the entry point
        ``name`` at ``precision``."""
        precision = normalize_precision(precision)
        if name in ("_regular_prec", "_gram_prec"):
            if precision not in _COMPUTE_CODES:
                raise ValueError(f"Unsupported floating-point precision: {precision}")
            route = native.ROUTE_FLOAT if name == "_regular_prec" else native.ROUTE_GRAM
            return route, _COMPUTE_CODES[precision], 16, precision, False
        if name == "_regular_i8":
            return native.ROUTE_INT8, native.F16, 16, "int8", self.fp16_first
        if precision in ("int8_bq", "int8"):
            return native.ROUTE_BQ_INT8, native.F16, 128, "int8", self.fp16_first
        if precision != "float8_e4m3fn":
            raise ValueError(f"Unsupported block-quantised precision: {precision}")
        return native.ROUTE_BQ_FP8, native.F16, 128, precision, False

    def _call(self, name, x, coeffs, eps, deterministic, precision, out, stats):
        route, compute, alignment, checked, fp16_first = self.call_spec(name, precision)
        return self._run(route, x, coeffs, eps, compute, alignment, checked, fp16_first, out, deterministic, stats)

    # Every entry point takes the reference's arguments plus two keyword-only extras: ``out``, a caller-owned
    # tensor for the result (the sharded step lets NS write straight into its gather buffer), and ``stats``,
    # the statistics partials that the momentum kernel left for ``x`` (then no pass over ``x`` is needed
    # for its norm).
    def _regular_prec(self, x, coeffs=None, eps=1e-7, deterministic=True, precision="float16", *, out=None, stats=None):
        """FP32 / BF16 / FP16 regular NS (src/i8muon/_cutlass_prec.py:90-106)."""
        return self._call("_regular_prec", x, coeffs, eps, deterministic, precision, out, stats)

    def _gram_prec(self, x, coeffs=None, eps=1e-7, deterministic=True, precision="float16", *, out=None, stats=None):
        """Gram-space NS with restarts given by I8MUON_GRAM_RESET (src/i8muon/_cutlass_prec.py:107-130)."""
        return self._call("_gram_prec", x, coeffs, eps, deterministic, precision, out, stats)

    def _regular_i8(self, x, coeffs=None, eps=1e-7, deterministic=True, precision="int8", *, block=False, out=None,
                    stats=None):
        """Global-scale INT8 NS, optionally after one FP16 iteration (src/i8muon/_cutlass.py:130-142)."""
        return self._call("_regular_bq" if block else "_regular_i8", x, coeffs, eps, deterministic, "int8", out, stats)

    # ------------------------------------------------ opt-in polynomial entry points
    def _regular_i8_factored(self, X, factor_rows, eps=1e-7, deterministic=True, *, out=None):
        """Completed-square rows ``(c, p, q)``: X <- c * ((G + p I)^2 + q I) X per row, all in the
        global-INT8 stages (the first row in FP16 when ``fp16_first``); src/i8muon/_cutlass.py:93-128."""
        factors = tuple(tuple(float(v) for v in row) for row in factor_rows)
        if not factors or any(len(row) != 3 or not all(map(math.isfinite, row)) for row in factors):
            raise ValueError("Expected nonempty finite (c,p,q) factor rows")
        return self._run(native.ROUTE_INT8_FACTORED, X, factors, eps, native.F16, 16, "int8", self.fp16_first, out,
                         deterministic)

    def _regular_i8_grouped_cubic(self, X, input_gain, cubic_gains, terminal_abc, eps=1e-7):
        """All-INT8 grouped cubics T <- -gain * (T T^T - I) T followed by one quintic; ignores
        ``fp16_first`` (src/i8muon/_cutlass.py:78-84, _cutlass_cubic.py:8-71)."""
        from .polynomial import grouped_cubic
        return grouped_cubic(self, X, input_gain, cubic_gains, terminal_abc, eps)

    def _regular_i8_cubic_abc(self, X, coeffs, eps=1e-7, deterministic=True, precision="int8"):
        """Saved cubic rows ``(a, b, 0)`` with a > 0 > b, then one terminal quintic row; all INT8
        (src/i8muon/_cutlass.py:86-91, _cutlass_cubic.py:74-87)."""
        if precision != "int8":
            raise ValueError("Cubic ABC evaluation requires INT8")
        from .polynomial import cubic_abc
        return cubic_abc(self, X, coeffs, eps)

    def _regular_bq(self, x, coeffs=None, eps=1e-7, deterministic=True, precision="float8_e4m3fn", *, out=None,
                    stats=None):
        """128x128 block-quantised NS: INT8 honours fp16_first, E4M3 never does
        (src/i8muon/_cutlass.py:71-76)."""
        if normalize_precision(precision) in ("int8_bq", "int8"):
            return self._regular_i8(x, coeffs, eps, deterministic, "int8", block=True, out=out, stats=stats)
        return self._call("_regular_bq", x, coeffs, eps, deterministic, precision, out, stats)


# What stands between a routed entry point and the library, as this file defines it.
_OWN_CODE = {name: CutlassNSInt8.__dict__[name] for name in (
    "_regular_prec", "_gram_prec", "_regular_i8", "_regular_bq", "_call", "_run", "call_spec")}


def runs_own_code(engine) -> bool:
    """Whether every entry point of ``engine`` does what this file says: no subclass, and nothing replaced on the
    class or on the object.  Only then may a caller go to the library without calling them."""
    return (type(engine) is CutlassNSInt8 and _OWN_CODE.keys().isdisjoint(engine.__dict__)
            and all(CutlassNSInt8.__dict__.get(name) is code for name, code in _OWN_CODE.items()))


def is_own_entry(engine, function) -> bool:
    """Whether ``function``, as the router returned it, is this engine's own entry point of that name."""
    code = _OWN_CODE.get(getattr(function, "__name__", None))
    return code is not None and getattr(function, "__self__", None) is engine and getattr(function, "__func__", None) is code


__all__ = ["CutlassNSInt8", "check_status", "status_word", "status_host", "post_status", "raise_if_reported"]
