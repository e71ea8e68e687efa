"""Compile the CUDA sources in this directory into ``pydtnn_b200/libb2c.so`` for sm_100a.

    python pydtnn_b200/csrc/build.py [--force] [-v] [--variant profile|switches]

Two development variants of the tensor-core kernel can be built next to the product library (never loaded by the
package):

* ``--variant profile``  -> ``pydtnn_b200/libb2c_profile.so`` (``-DB2C_TC_PROFILE``): every warp role of CTA 0 adds up
  the cycles it spends waiting and working (a slot per ``TC_PROF_ADD``), read with ``b2c_debug_prof``.
* ``--variant switches`` -> ``pydtnn_b200/libb2c_switches.so`` (``-DB2C_TC_SWITCHES``): the environment variable
  ``B2C_TC_DBG`` switches parts of the kernel off to see what the rest costs (results are then wrong): 2 = one MMA of
  three, 4 = transform warps do no work, 32 = no MMA, 64 = no TMA loads; values add.
"""
import os
import re
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
SOURCES = ["api.cu", "conv_fma.cu", "conv_tc.cu", "fc_mma.cu", "aux_ops.cu"]
OUT = os.path.join(PKG, "libb2c.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v"]
VARIANTS = {None: ("", [], OUT),
            "profile": (".profile", ["-DB2C_TC_PROFILE"], os.path.join(PKG, "libb2c_profile.so")),
            "switches": (".switches", ["-DB2C_TC_SWITCHES"], os.path.join(PKG, "libb2c_switches.so"))}

# conv_tc_kernel<MODE, BN, STAGES, SK, SLABS, BSRC, STREAM, MULTI, RESKB, FINE, BOTH, PAIR> in a symbol
_TC_KERNEL = re.compile(r"Compiling entry function '\w*conv_tc_kernelI" + "".join(f"L[ib](?P<{a}>\\d+)E" for a in
                        ("mode", "bn", "stages", "sk", "slabs", "bsrc", "stream", "multi", "reskb", "fine", "both")) + r"(?:Lb\d+E)?E.*?Used (?P<regs>\d+) registers", re.S)
LAUNCH_REGISTERS = 128


def check_role_registers(ptxas_output):
    """The warp roles of the kernels with warps of their own for the B tile (``tc_b_warps``) share out 4 x 128 registers: a variant
    that was compiled to fewer would wait for registers that never come, so it must not be linked (its launch is refused)."""
    found = 0
    for m in _TC_KERNEL.finditer(ptxas_output):
        v = {k: int(x) for k, x in m.groupdict().items()}
        if (v["mode"] == 1 or v["bsrc"] != 0) and v["reskb"] == 0 and v["stream"] != 2 and not v["both"]:
            found += 1
            if v["regs"] != LAUNCH_REGISTERS:
                raise RuntimeError(f"conv_tc_kernel with {LAUNCH_REGISTERS} registers a thread to share out was compiled to {v['regs']}: {v}")
    return found


def build(force=False, verbose=False, variant=None):
    suffix, defines, out = VARIANTS[variant]
    srcs = [os.path.join(HERE, s) for s in SOURCES]
    deps = srcs + [os.path.join(HERE, "b2c_common.cuh"), os.path.join(os.path.dirname(PKG), "include", "b2c.h")]
    deps += [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith(".cuh")]
    if not force and os.path.exists(out) and all(os.path.getmtime(d) <= os.path.getmtime(out) for d in deps):
        return out
    objs = []
    procs = []
    for s in srcs:
        o = s[:-3] + suffix + ".o"
        objs.append(o)
        procs.append((s, subprocess.Popen([NVCC, *FLAGS, *defines, "-c", s, "-o", o], stdout=subprocess.PIPE,
                                          stderr=subprocess.STDOUT, text=True)))
    failed = False
    for s, p in procs:
        text, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(text)
        if p.returncode:
            failed = True
        elif os.path.basename(s) == "conv_tc.cu" and not check_role_registers(text):
            raise RuntimeError("no conv_tc_kernel found in what ptxas says")
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.run([NVCC, "-shared", "-o", out, *objs, "-gencode", "arch=compute_100a,code=sm_100a"], check=True)
    return out


if __name__ == "__main__":
    variant = sys.argv[sys.argv.index("--variant") + 1] if "--variant" in sys.argv else None
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, variant=variant))
