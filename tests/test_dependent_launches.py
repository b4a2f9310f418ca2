"""The rules a kernel keeps that may start while the kernel before it still runs: checks on the sources, and of the call that launches it."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sptorch_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _block(text, at):
    """The braces' contents that open at text[at]."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError("unbalanced braces")


def _kernels(name):
    """[(kernel, parameter list, body)] of the file's kernels that wait for their predecessor themselves."""
    text, out = _source(name), []
    for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\s*\(([^{]*?)\)\s*\{", text):
        body = _block(text, m.end() - 1)
        if "pdl_acquire()" in body:
            out.append((m.group(1), m.group(2), body))
    return out


def test_row_operations_read_nothing_ahead_of_the_wait():
    """These kernels serve the public operations as well as the models: any operand, norm weights included, may be what the kernel before
    has just written."""
    kernels = _kernels("rowops.cu") + _kernels("rope.cu")
    assert len(kernels) >= 6
    for kernel, params, body in kernels:
        pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", params)
        ahead = body[:body.index("pdl_acquire()")]
        for p in set(pointers) - {"status"}:
            assert not re.search(r"(?<![.\w])%s\b" % p, ahead), f"{kernel} reads {p} ahead of its wait"


# what a model's parameters, tables and per-step device words are called in the kernels: written before the step's first launch
SETTLED = {"gamma", "beta", "gamma2", "bias", "bias2", "w", "w2", "W", "a2", "head_norm", "conv", "temp", "cs", "denom", "rope", "table", "side_table",
           "ids", "state", "offset_dev", "slopes", "sched", "sp"}
# files whose kernels serve public operations too, where norm weights and biases are operands like any other
OPERATIONS = {"rowops.cu": SETTLED - {"gamma", "beta", "w", "bias"}, "gemm.cu": SETTLED - {"bias"}, "rope.cu": SETTLED, "attention_fused.cu": SETTLED}


def _arguments(text, call):
    for m in re.finditer(r"\b%s\s*\(" % call, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_what_a_predecessor_writes_is_not_read_as_constant():
    """A kernel that starts early lives while its predecessor still writes: read-only loads and const __restrict__ pointers are for what is
    settled before the step's first launch."""
    files = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "pdl.cuh" in open(os.path.join(CSRC, f)).read())
    seen = 0
    for f in files:
        allowed = OPERATIONS.get(f, SETTLED)
        for kernel, params, body in _kernels(f):
            seen += 1
            for name in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params):
                assert name in allowed, f"{f}: {kernel} takes {name} as constant"
            for call in ("__ldg", "__ldcs", "__ldca", "__ldcg"):
                for arg in _arguments(body, call):
                    assert set(re.findall(r"(?<!\w)(?:\w+\.)*(\w+)", arg)) & allowed, f"{f}: {kernel} reads {arg!r} with {call}"
    assert seen >= 25
    # helpers of those kernels
    helpers = _source("gla.cu")
    assert "__ldg" not in helpers[helpers.index("struct TileLoad"):helpers.index("__global__", helpers.index("struct TileLoad"))]
    vec = _source("rowops.cu")
    assert "__ldcs" not in vec[:vec.index("row_reduce")]


def test_aligned_cluster_barriers_come_behind_a_warp_barrier():
    """Lanes that a branch has parted must not reach an aligned barrier one by one: the two helpers bring the warp together, and nothing else
    issues the instruction."""
    for f in sorted(os.listdir(CSRC)):
        lines = [ln for ln in _source(f).splitlines() if "barrier.cluster" in ln and ".aligned" in ln] if f.endswith((".cu", ".cuh", ".h")) else []
        for ln in lines:
            assert f == "sm100.cuh" and 0 <= ln.find("__syncwarp()") < ln.find("barrier.cluster"), f"{f}: {ln.strip()}"
        assert f != "sm100.cuh" or len(lines) == 2


def test_streaming_linear_leaves_a_wait_by_warps():
    """Behind these two waits come instructions of the whole warp (elect, tcgen05.ld): lanes of which one gave up must not part."""
    waits = re.findall(r"\b(mbar_wait\w*)\(([^;]*)\);", _source("linear_stream.cu"))
    assert len(waits) == 3
    for call, args in waits:
        assert call == ("mbar_wait" if "kErrProducerWait" in args else "mbar_wait_warp"), args      # the producer is one lane


def test_vector_accesses_of_shared_arrays_find_them_aligned():
    """An array of scalars is promised the alignment of one scalar, wherever the compiler happens to place it: what is read or written eight or sixteen
    bytes at a time says so in its declaration."""
    wide = r"(?:u?int|float)[24]|uint64_t|__nv_bfloat162"
    for f in sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))):
        text = _source(f)
        for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\s*\(([^{]*?)\)\s*\{", text):
            body = _block(text, m.end() - 1)
            narrow = set()
            for aligned, kind, names in re.findall(r"(?<!extern )__shared__ (__align__\(\d+\) )?(?:volatile )?([\w:]+) ([^;]*);", body):
                if not aligned and not re.fullmatch(wide, kind):
                    narrow |= set(re.findall(r"(\w+)\[", names))
            for _ in range(4):                                               # pointers into them, and pointers made of those
                narrow |= {to for to, of in re.findall(r"\*\s*(?:const )?(\w+)\s*=\s*&?(\w+)\b", body) if of in narrow}
            for kind, name in re.findall(r"reinterpret_cast<(?:const )?(%s)\s*\*>\(\s*&?(\w+)" % wide, body):
                assert name not in narrow, f"{f}: {m.group(1)} takes {name} as {kind}"


def test_a_cluster_sends_only_to_ctas_that_are_there():
    """Asynchronous stores are counted on the receiver's barrier.  A receiver that gave up waiting for them may not leave while others still send:
    it meets them at the cluster's barrier, whose arrival is theirs on leaving at the latest, and lets what is on its way land."""
    merge = _source("decode.cu")
    merge = _block(merge, merge.index("{", merge.index("void merge_parts")))
    wait = re.search(r"if \(!sm100::mbar_wait_warp\([^;]*\)\s*\{", merge)
    assert wait and merge.index("send4(") < wait.start() and "mbar_wait<" not in merge
    given_up = _block(merge, wait.end() - 1)
    assert 0 <= given_up.find("cluster_sync()") < given_up.find("globaltimer() - t0") < given_up.find("return")
    stream = _source("linear_stream.cu")
    sends = stream.rindex("send16(")
    assert sends < stream.index("cluster_arrive_relaxed()", sends) < stream.index("cluster_wait()", sends) < stream.index("if (abort_flag)", sends) < stream.index("globaltimer() - t0", sends)
    senders = {f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and re.search(r"\bsend(?:4|16)\(|st\.async", _source(f))}
    assert senders == {"sm100.cuh", "decode.cu", "linear_stream.cu"}


def test_short_attention_stores_its_columns_over_all_banks():
    """Keys and queries are brought by rows and stored by columns: at every step of a warp the 32 words it stores lie in 32 banks, and it brings every
    piece of four values of every row once, sixteen rows' whole sectors at a time."""
    text = _source("attention.cu")
    row, column = re.search(r"auto piece = .*?\br = ([^;]*); c = ([^;]*);", text).groups()
    row, column = row.replace("/", "//"), column.replace("/", "//")
    for rows in (32, 64):
        for vecs in (1, 2, 8, 9, 16, 32):
            brought = set()
            for first in range(0, rows * (vecs + 1) // 2 * 2, 32):
                lanes = [(eval(row, {}, {"i": i, "rows": rows}), eval(column, {}, {"i": i, "rows": rows})) for i in range(first, first + 32)]
                assert len({(c * (rows + 4) + r) % 32 for r, c in lanes}) == 32
                assert len({(r, c // 8) for r, c in lanes}) == 16
                brought |= {(r, c) for r, c in lanes if c < 4 * vecs}
            assert brought == {(r, 4 * v) for r in range(rows) for v in range(vecs)}


def test_tensor_memory_is_taken_before_the_next_launch_may_start():
    """tcgen05.alloc waits without a limit; it ends because a later grid cannot hold columns that an earlier one still asks for."""
    seen = []
    for f in sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")):
        for kernel, _, body in _kernels(f):
            if "tmem_alloc" in body:
                seen.append(kernel)
                assert body.rindex("tmem_alloc") < body.index("pdl_release()"), f"{f}: {kernel}"
    assert len(seen) == 3, seen


def test_decode_attention_is_held_to_the_ctas_its_rule_counts_on(tmp_path):
    """The rule that splits a cache over CTAs counts how many of them the SMs hold at once: the registers that the compiler gives each kernel must
    leave room for as many."""
    held = {("mma", 2, 1, 4): 6, ("mma", 2, 1, 8): 2, ("mma", 2, 1, 16): 1, ("mma", 4, 2, 4): 3, ("mma", 4, 2, 8): 1, ("f", 4): 6, ("f", 16): 1, ("13__nv_bfloat16", 4): 6,
            ("13__nv_bfloat16", 16): 1}
    cmd = ["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xptxas", "-v", "-c",
           os.path.join(CSRC, "decode.cu"), "-o", str(tmp_path / "decode.o")]
    log = subprocess.run(cmd, capture_output=True, text=True, check=True, timeout=300).stderr
    seen = {}
    for name, registers in re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", log, re.S):
        kernel = re.search(r"attention_last_token_(?:mma|rows)_kernelI(f|13__nv_bfloat16)?((?:Li\d+E)+)E", name)
        if kernel:
            seen[(kernel.group(1) or "mma", *map(int, re.findall(r"\d+", kernel.group(2))))] = int(registers)
    assert set(seen) == set(held)
    for k, registers in seen.items():
        assert 65536 // (-(-registers // 8) * 8 * 32 * k[-1]) >= held[k], f"{k}: {registers} registers"


_REFUSED = """
#include "common.h"
#include <stdio.h>
namespace spt { Runtime& rt() { static Runtime r; return r; } }
__global__ void nothing_kernel(int) {}
int main() {
    const cudaError_t good = spt::launch_dependent(nothing_kernel, dim3(1), dim3(1), 0, true, 1, 0);
    const cudaError_t none = spt::launch_dependent(nothing_kernel, dim3(0), dim3(1), 0, true, 1, 0);
    const cudaError_t last = cudaPeekAtLastError();
    printf("%d %d %d %d\\n", good == cudaSuccess, none == cudaErrorInvalidConfiguration, last == cudaSuccess, cudaDeviceSynchronize() == cudaSuccess);
}
"""


@pytest.mark.gpu
def test_a_refused_launch_leaves_no_error_for_the_next_one(tmp_path):
    """A launch that the runtime refuses (an empty grid) reports it itself; the last error, which ordinary launches are checked by, must not hand
    it on to the next one."""
    (tmp_path / "refused.cu").write_text(_REFUSED)
    exe = str(tmp_path / "refused")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, str(tmp_path / "refused.cu"), "-o", exe], check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.stdout.split() == ["1"] * 4, out.stdout + out.stderr
