"""ctypes.pythonapi is one object for the whole process: importing the package
leaves the prototypes that another library may have set there as they were."""

import subprocess
import sys

CHECK = """
import ctypes
names = ("PyBytes_FromStringAndSize", "PyBytes_AsString")
before = [(getattr(ctypes.pythonapi, n).restype, getattr(ctypes.pythonapi, n).argtypes) for n in names]
import rivet_prores_b200
assert [(getattr(ctypes.pythonapi, n).restype, getattr(ctypes.pythonapi, n).argtypes) for n in names] == before
"""


def test_importing_leaves_the_shared_prototypes_alone():
    r = subprocess.run([sys.executable, "-c", CHECK], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
