"""What the memory model asks of the kernels and no run can be relied on to show, read from their sources."""
import ctypes
import glob
import os
import re
import shutil
import subprocess

import pytest

import picotron_b200

CSRC = os.path.join(os.path.dirname(picotron_b200.__file__), "csrc")
TOKENS = re.compile(r"[{}]|mbar_wait\(|tcgen05_fence_after\(\)|(?:tmem_(?:ld|st)_32x32b|umma_bf16)\w*\(")


def unfenced_accesses(src):
    """Lines of tensor-memory accesses and MMAs that follow an mbarrier wait without tcgen05.fence::after_thread_sync on every
    way between the two (a fence in a block that is entered conditionally counts inside that block only)."""
    src = re.sub(r"//[^\n]*", "", src)
    depth, waits, fences, found = 0, [], [], []      # waits: depths of those not fenced yet; fences: depths of conditional fences
    for m in TOKENS.finditer(src):
        token = m.group(0)
        if token == "{":
            depth += 1
        elif token == "}":
            depth -= 1
            fences = [f for f in fences if f <= depth]
        elif token == "mbar_wait(":
            statement = src[max(src.rfind(c, 0, m.start()) for c in ";{}"):m.start()]
            # `if (ok && mbar_wait(..)) {`: what depends on the wait stands in the block that follows
            waits.append(depth + (1 if "if" in statement and not statement.rstrip().endswith("!") else 0))
            fences = []
        elif token.startswith("tcgen05_fence"):
            waits = [w for w in waits if w < depth]
            if waits:
                fences.append(depth)
        elif waits and not fences:
            found.append(src.count("\n", 0, m.start()) + 1)
    return found


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*tcgen05.cu"))), ids=os.path.basename)
def test_tensor_memory_is_fenced_after_every_wait(path):
    with open(path) as f:
        assert unfenced_accesses(f.read()) == []


def test_the_check_sees_a_missing_and_a_conditional_fence():
    wait = "if (!mbar_wait(&b, 0, a)) { break; }\n"
    assert unfenced_accesses(wait + "tcgen05_fence_after();\ntmem_st_32x32b_x32(t, r);") == []
    assert unfenced_accesses(wait + "tmem_st_32x32b_x32(t, r);") == [2]
    assert unfenced_accesses(wait + "if (m) { tcgen05_fence_after(); tmem_ld_32x32b_x32(t, r); }\ntmem_st_32x32b_x32(t, r);") == [3]
    assert unfenced_accesses("if (ok && mbar_wait(&b, 0, a)) {\ntcgen05_fence_after();\ntmem_ld_32x32b_x32(t, r); }") == []


def test_a_build_with_other_register_counts_than_a_kernel_depends_on_fails():
    from picotron_b200 import build
    log = ("ptxas info    : Compiling entry function '_ZN2pt4attn15attn_bwd_kernelILi64ELb0ELb0EEEv' for 'sm_100a'\n"
           "ptxas info    : Function properties for _ZN2pt4attn15attn_bwd_kernelILi64ELb0ELb0EEEv\n"
           "    0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads\n"
           "ptxas info    : Used {} registers, used 1 barriers\n"
           "ptxas info    : Compiling entry function '_Z10add_kernel' for 'sm_100a'\n"
           "ptxas info    : Used 32 registers\n")
    build.check_registers(log.format(128))
    with pytest.raises(RuntimeError, match="attn_bwd_kernel.*126 registers"):
        build.check_registers(log.format(126))
    with open(os.path.join(CSRC, "attention_tcgen05.cu")) as f:
        assert f"BWD_REGS = {build.FIXED_REGISTERS['attn_bwd_kernel']}," in f.read()


PER_DEVICE_PROBE = r"""
#include "per_device.h"
static pt::PerDevice state;
extern "C" int get(int device, int result, int* calls) {
  return state.get(device, [&] { ++*calls; return result; });
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_launcher_state_is_found_once_on_every_device_and_a_failure_is_not_kept(tmp_path):
    src, lib = tmp_path / "probe.cpp", tmp_path / "probe.so"
    src.write_text(PER_DEVICE_PROBE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    probe, calls = ctypes.CDLL(str(lib)), ctypes.c_int(0)

    def get(device, result):
        return probe.get(device, result, ctypes.byref(calls)), calls.value

    assert get(0, 7) == (7, 1) and get(0, 9) == (7, 1)           # kept
    assert get(1, -3) == (-3, 2) and get(1, 5) == (5, 3) and get(1, 6) == (5, 3)
    assert get(63, 1) == (1, 4) and get(0, 9) == (7, 4)
    assert get(64, 2) == (2, 5) and get(-1, 2) == (2, 6)         # beyond the table: found at every call


@pytest.mark.parametrize("name", ["elementwise.cu", "gemm_tcgen05.cu", "gemm_pair_tcgen05.cu", "gemm_allreduce_tcgen05.cu", "attention_tcgen05.cu"])
def test_kernel_attributes_are_set_on_every_device(name):
    """What remembers that a kernel's attribute was set is kept per device: the attribute is that of the current device alone."""
    with open(os.path.join(CSRC, name)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    keeper = None
    for m in re.finditer(r"static (?:const )?(\w+) \w+(?: =|;)|cudaFuncSetAttribute", src):
        if m.group(0) == "cudaFuncSetAttribute":
            assert keeper == "PerDevice", src[m.start() - 200:m.start() + 100]
        else:
            keeper = m.group(1)
