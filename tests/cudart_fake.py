"""Runs a scenario of a test file in a child process whose CUDA runtime calls can
be made to fail (drivers/cudart_fake.c, preloaded there).  Nothing fails on the
GPU: a faked call returns its error on the host and does not happen."""
import ctypes
import os
import subprocess
import sys

INSTANTIATE, GRAPH_LAUNCH, COOPERATIVE, ALLOCATION = range(4)

HERE = os.path.dirname(os.path.abspath(__file__))


def run(test_file, scenario, tmp_path, *args):
    """`python test_file scenario args...` in a child with the fakes preloaded."""
    lib = str(tmp_path / "cudart_fake.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", f"-I{cuda}/include", os.path.join(HERE, "drivers", "cudart_fake.c"),
                    "-o", lib, "-ldl"], check=True)
    r = subprocess.run([sys.executable, test_file, scenario, *map(str, args)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=lib))
    assert r.returncode == 0, r.stdout + r.stderr


def main(scenarios):
    """In the child: the scenario named on the command line, given the package, its scenes and the fakes."""
    if HERE not in sys.path:
        sys.path.insert(0, HERE)
    from conftest import load_package
    ds = load_package()
    import dem_sphsource_gb300.scenes as scenes
    fakes = ctypes.CDLL(None)
    fakes.fake_arm.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_size_t]
    fakes.fake_count.restype = ctypes.c_longlong
    scenarios[sys.argv[1]](ds, scenes, fakes, *sys.argv[2:])
