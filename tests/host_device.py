"""The device headers of pyclaw_b200/csrc compiled for the host, for tests that
look at them without a GPU: a copy of the headers with their inline PTX replaced
(the few instructions that matter by C++, the others by nothing), against the
stand-in tests/host_cuda/cuda_runtime.h."""
import os
import re
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pyclaw_b200", "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
PTX = {"rcp.approx.ftz.f64": "r = emu::rcp_seed(y);", "rsqrt.approx.ftz.f64": "y = emu::rsqrt_seed(x);",
       "atom.add.acq_rel.gpu.global.u32": "arrived = __atomic_fetch_add(a.ticket, 1u, __ATOMIC_ACQ_REL);"}


def without_ptx(text):
    """text with every asm statement replaced as PTX says, by an empty statement otherwise"""
    out, at = [], 0
    for m in re.finditer(r"\basm(?:\s+volatile)?\s*\(", text):
        end, depth, quoted = m.end(), 1, False
        while depth:
            c = text[end]
            if c == '"' and text[end - 1] != "\\":
                quoted = not quoted
            if not quoted:
                depth += (c == "(") - (c == ")")
            end += 1
        stmt = text[m.start():end]
        out += [text[at:m.start()], next((v[:-1] for k, v in PTX.items() if k in stmt), "(void)0")]
        at = end
    return "".join(out) + text[at:]


def compile_host(source, folder, shared=True, flags=()):
    """source (C++ text that includes the headers by name) -> path of the shared
    object (or program) built from it in folder"""
    inc = os.path.join(str(folder), "pyclaw_b200", "csrc")
    os.makedirs(inc)
    shutil.copytree(INCLUDE, os.path.join(str(folder), "include"))
    for name in os.listdir(CSRC):
        if name.endswith((".cuh", ".h")):
            with open(os.path.join(CSRC, name)) as f, open(os.path.join(inc, name), "w") as g:
                g.write(without_ptx(f.read()))
    src, out = os.path.join(str(folder), "host.cpp"), os.path.join(str(folder), "host.so" if shared else "host")
    with open(src, "w") as f:
        f.write(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-mfma", "-ffp-contract=off", "-pthread", "-w",
                    "-I", os.path.join(HERE, "host_cuda"), "-I", inc] + (["-shared", "-fPIC"] if shared else []) +
                   list(flags) + ["-o", out, src], check=True)
    return out
