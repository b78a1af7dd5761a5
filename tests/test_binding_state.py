"""Importing the binding changes nothing that other code in the process shares."""
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parents[1] / "rust-sloth_gb300"


def test_pythonapi_prototypes_stay_as_they_were():
    code = (f"import ctypes, sys; sys.path.insert(0, {str(PKG)!r}); f = ctypes.pythonapi.PyBytes_FromStringAndSize; "
            "before = (f.argtypes, f.restype); import sloth_gpu as S; assert (f.argtypes, f.restype) == before, "
            "(f.argtypes, f.restype); b = S._new_bytes(None, 5); assert type(b) is bytes and len(b) == 5")
    subprocess.run([sys.executable, "-c", code], check=True)
