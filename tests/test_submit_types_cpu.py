"""An op list is bytes: anything else is refused before the library is called (CPU only)."""
import numpy as np
import pytest

from pixels_gb300 import _lib
from pixels_gb300.ir import Program


@pytest.mark.parametrize("convert", [bytearray, memoryview, list, lambda b: np.frombuffer(b, np.uint8), lambda b: len(b),
                                     lambda b: b.decode("latin-1"), lambda b: None])
def test_only_bytes(built_lib, convert):
    ir = Program().to_bytes()
    with pytest.raises(TypeError):
        _lib.submit_ops(None, convert(ir))
    with pytest.raises(_lib.PxError):  # bytes reach the library, which refuses the handle
        _lib.submit_ops(None, ir)
