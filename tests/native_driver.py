"""C++ programs of the tests, compiled against the engine's own headers and
linked to libhfx.so: host code that has no entry point of its own."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB_DIR = os.path.join(REPO, "hartree_fock_cpp_gb300")
INCLUDE = ["-I", os.path.join(LIB_DIR, "csrc"), "-I", os.path.join(REPO, "include"), "-I", "/usr/local/cuda/include"]


def compile_driver(source, path, link=True):
    """Build `source` to the executable `path` (link=False: to an object);
    returns the compiler's result."""
    src = str(path) + ".cpp"
    with open(src, "w") as f:
        f.write(source)
    cmd = ["g++", "-std=c++17", "-O1", "-o", str(path), src] + INCLUDE
    cmd += ["-L", LIB_DIR, "-lhfx", "-Wl,-rpath," + LIB_DIR, "-Wl,--allow-shlib-undefined", "-lpthread"] if link else ["-c"]
    return subprocess.run(cmd, capture_output=True, text=True)


def run_program(path, *args, stdin=None):
    """The standard output of a built program."""
    r = subprocess.run([str(path)] + [str(a) for a in args], capture_output=True, text=True, timeout=300, input=stdin)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def run_driver(source, path, *args):
    """Build and run; the program's standard output."""
    c = compile_driver(source, path)
    assert c.returncode == 0, c.stderr
    return run_program(path, *args)
