"""Compile the CUDA sources in `csrc/` into `libturbot5_b200.so`, and the native host side in
`csrc/host/` into the Python extension `_host.so`, next to this file.

    python -m turbot5_b200.build [--force]

The library is built for sm_100a only, in-tree, with nvcc (no JIT cache; its ABI is plain C, see
include/turbot5_b200.h).  The extension is plain C++ over the library's C ABI and PyTorch's C++ API:
argument checks, allocation, autograd nodes and the launch sequences of whole passes.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libturbot5_b200.so")
SOURCES = ["api.cu", "bucket.cu", "attn_fwd_sm100.cu", "attn_fwd2_sm100.cu", "attn_bwd_sm100.cu", "attn_fwd_simt.cu", "attn_bwd_simt.cu", "decode.cu", "decoder_step.cu",
           "rmsnorm.cu", "padding.cu", "fused_ops.cu"]
HOST = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(HERE, "_host.so")
HOST_SOURCES = ["ops.cpp", "stack.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _newest(folder):
    files = [os.path.join(folder, f) for f in os.listdir(folder) if f.endswith((".cu", ".cuh", ".cpp", ".h"))]
    files.append(os.path.join(os.path.dirname(HERE), "include", "turbot5_b200.h"))
    return max(os.path.getmtime(f) for f in files)


def _stale(target, folder):
    return not os.path.exists(target) or os.path.getmtime(target) < _newest(folder)


def _run_all(commands, verbose):
    """Run (source, command) pairs in parallel; returns {source: compiler output}."""
    procs = [(src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)) for src, cmd in commands]
    logs = {}
    for src, pr in procs:
        out, _ = pr.communicate()
        logs[src] = out.decode()
        if verbose and out:
            sys.stderr.write(logs[src])
    for src, pr in procs:
        if pr.returncode != 0:
            raise RuntimeError(f"compiling {src} failed:\n{logs[src]}")
    return logs


def _host_flags():
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "/usr/local/cuda/include", sysconfig.get_paths()["include"]]
    compile_flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", *("-I" + i for i in inc)]
    link_flags = ["-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10",
                  "-lc10_cuda", "-L/usr/local/cuda/lib64", "-lcudart", "-lcublas", "-L" + HERE, "-l:libturbot5_b200.so",
                  "-Wl,-rpath,$ORIGIN"]
    return compile_flags, link_flags


def _link(cmd, target):
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout.decode())
    os.replace(target + ".tmp", target)


def build(force: bool = False, verbose: bool = False) -> str:
    """Build the shared library and the host extension if they are missing or older than their sources."""
    cuda, host = force or _stale(LIB, CSRC), force or _stale(HOST_LIB, HOST)
    commands, objs, host_objs = [], [], []
    if cuda:
        for src in SOURCES:
            objs.append(os.path.join(CSRC, src.replace(".cu", ".o")))
            commands.append((src, [_nvcc(), "-Xptxas=-v", *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", objs[-1]]))
    if host:
        compile_flags, link_flags = _host_flags()
        for src in HOST_SOURCES:
            host_objs.append(os.path.join(HOST, src.replace(".cpp", ".o")))
            commands.append((src, ["g++", *compile_flags, "-c", os.path.join(HOST, src), "-o", host_objs[-1]]))
    logs = _run_all(commands, verbose)
    if cuda:
        for src in SOURCES:
            with open(_ptxas_log(src), "w") as f:      # registers and spills per kernel, see resource_report()
                f.write(logs[src])
        _link([_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB + ".tmp", *objs], LIB)
    if host:
        _link(["g++", "-shared", "-o", HOST_LIB + ".tmp", *host_objs, *link_flags], HOST_LIB)
    return LIB


def _ptxas_log(src: str) -> str:
    return os.path.join(CSRC, src.replace(".cu", ".ptxas.txt"))


def resource_report(src: str) -> dict:
    """{mangled kernel name: {"registers", "spill_stores", "spill_loads", "stack"}} from ptxas's own
    report for one source file (written by `build`; compiled again here, without an object file, when
    the library was built by an older copy of this script).  A few extra live values in a softmax loop
    can turn into spills that cost a kernel 15 % without failing any test, so the tests hold the hot
    kernels to a budget."""
    import re
    log = _ptxas_log(src)
    if not os.path.exists(log) or os.path.getmtime(log) < os.path.getmtime(os.path.join(CSRC, src)):
        cmd = [_nvcc(), "-Xptxas=-v", *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", os.devnull]
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout.decode()}")
        with open(log, "w") as f:
            f.write(r.stdout.decode())
    report, name = {}, None
    for line in open(log):
        m = re.search(r"Compiling entry function '([^']+)'", line)
        if m:
            name = m.group(1)
            report[name] = {"registers": 0, "spill_stores": 0, "spill_loads": 0, "stack": 0}
            continue
        if name is None:
            continue
        m = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m:
            report[name].update(stack=int(m.group(1)), spill_stores=int(m.group(2)), spill_loads=int(m.group(3)))
        m = re.search(r"Used (\d+) registers", line)
        if m:
            report[name]["registers"] = int(m.group(1))
    return report


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
