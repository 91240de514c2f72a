"""Lower limits of the fused steps of a context or a batch (score_internal_step_limits), so that small domains take every path."""
import ctypes as C

from score_gb300 import _abi


class StepLimits(C.Structure):
    _fields_ = [("host_polls", C.c_uint32), ("group_polls", C.c_uint32), ("wide", C.c_uint32), ("block_slots", C.c_uint32),
                ("slots", C.c_uint64), ("number", C.c_uint32),
                ("refuse_after", C.c_uint32), ("stage", C.c_uint64)]


def set_limits(owner, **kw):
    """owner: GrowthMachine or Batch; what is not named keeps its default.  number: the next command's step number;
    refuse_after: cooperative launches until one is refused; stage: bytes beyond which a staging buffer is refused."""
    f = _abi.load().score_internal_step_limits
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_void_p, C.POINTER(StepLimits)]
    lim = StepLimits(**{**{n: 2 ** (8 * C.sizeof(t)) - 1 for n, t in StepLimits._fields_}, "number": 0, **kw})
    assert f(getattr(owner, "_ctx", None), getattr(owner, "_b", None), C.byref(lim)) == _abi.OK
