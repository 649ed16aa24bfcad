"""Order of a kernel's ring buffers, from the waits in its source: a slot is read before it is filled again."""
import os
import re
import subprocess

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc", "kernels", "gemm_fp8_block.cu")


def test_scales_of_few_rows_are_read_before_their_slot_is_filled_again():
    """The events of a CTA of the FP8 product of few rows (copy of a block's scales, MMA, hand-back of its accumulator, reading of its
    scales) and what each waits for.  A warp that is held up before it reads must not find the scales of a later block."""
    text = open(SRC).read()
    cfg = text[text.index("struct FrCfg"):]
    stages, nbuf, slots = [int(re.search(rf"\b{n} = (\d+)", cfg).group(1)) for n in ("STAGES", "NBUF", "SA_SLOTS")]
    body = text[text.index("gemm_fp8_rows_kernel("):]
    back_first = body.index("mbar_arrive(&part_empty") < body.index("= sa[")      # the accumulator is handed back before the scales are read
    n, before = 4 * slots, {}
    for i in range(n):
        before["copy", i] = [("copy", i - 1), ("mma", i - stages)]                # the operand stage is free
        before["mma", i] = [("mma", i - 1), ("copy", i), ("back", i - nbuf)]
        first, second = ("back", "read") if back_first else ("read", "back")
        before[first, i] = [("mma", i), (second, i - 1)]
        before[second, i] = [(first, i)]

    def earlier(event):
        seen, todo = set(), [event]
        while todo:
            for e in before.get(todo.pop(), []):
                if e[1] >= 0 and e not in seen:
                    seen.add(e)
                    todo.append(e)
        return seen
    for i in range(slots, n):
        assert ("read", i - slots) in earlier(("copy", i)), f"block {i} overwrites scales that may not have been read"


def test_few_rows_ctas_leave_after_their_copies_and_their_peers():
    """After a wait that ran out, too: behind the last access to a peer's memory, and before a CTA gives up its own, it waits for the
    copies that it has started and for the peers."""
    text = open(SRC).read()
    body = text[text.index("gemm_fp8_rows_kernel("):]
    body = body[:body.index("\n}\n")]
    end = body[body.rindex("mbar_arrive_remote("):]
    order = [end.index(s) for s in ("__syncthreads();", "if (threadIdx.x == 0 && *abort_flag)", "mbar_wait(&full[", "mbar_wait(&sa_full[",
                                    "cluster_arrive();", "cluster_wait();", "tmem_dealloc(")]
    assert order == sorted(order)


def _kernels():
    """(name, body) of every kernel."""
    folder = os.path.dirname(SRC)
    for f in sorted(os.listdir(folder)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(folder, f)).read())
        for part in re.split(r"__global__ ", text)[1:]:
            body = part[:part.index("\n}\n") + 3]
            yield f + ": " + re.search(r"(\w+)\s*\((?!\()(?:[^()]|\([^()]*\))*\)\s*\{", body[body.index("void"):]).group(1), body


def test_dependents_may_start_when_tensor_memory_is_allocated():
    """The successor of a kernel may become resident beside it and take tensor memory, which it holds until this kernel has completed: each
    CTA has its own before it lets the successor start."""
    seen = 0
    for name, body in _kernels():
        if "tmem_alloc" in body and "pdl_trigger" in body:
            seen += 1
            between = body[body.index("tmem_alloc"):body.index("pdl_trigger")] if body.index("tmem_alloc") < body.index("pdl_trigger") else ""
            assert "__syncthreads();" in between, name
    assert seen >= 8


def test_scales_of_a_pair_are_handed_back_by_the_warps_that_read_them():
    """FP8 product on CTA pairs: a slot of the scales' ring is filled again when every epilogue warp of the same CTA has released it, behind
    its last access.  (Handing back an accumulator orders tensor memory alone, and goes to the other CTA.)"""
    text = open(os.path.join(os.path.dirname(SRC), "gemm_fp8_pair.cu")).read()
    body = re.sub(r"//[^\n]*", "", text[text.index("gemm_fp8_pair_kernel("):])
    assert "mbar_init(&sa_empty[i], Cfg::EPI)" in body
    fill, read = body[body.index("if (warp == 0)"):body.index("else if (warp == 1)")], body[body.index("float acc[32];"):]
    wait = fill.index("if (gb >= SLOTS && !mbar_wait(&sa_empty[gb % SLOTS], (gb / SLOTS - 1) & 1,")
    assert wait < fill.index("mbar_expect_tx(") and wait < fill.index("tma_load_2d_pair(sSA")
    after = read[read.index("= sa[j];"):]
    assert after.index("__syncwarp();") < after.index("mbar_arrive(&sa_empty[slot]") < after.index("finish")
    assert read.count("sa[j]") == 1


def test_programmatic_launch_has_one_switch(tmp_path):
    """BLAZE_PDL: unset, the products on CTA pairs alone start before their predecessor has finished; 0, nothing does; 1, all may.  Every
    launch with the attribute asks."""
    prog = tmp_path / "level.cpp"
    prog.write_text('#include "blaze/host.h"\n#include <stdio.h>\nint main() { printf("%d %d", blz::pdl_pairs(), blz::pdl_enabled()); }\n')
    root = os.path.dirname(os.path.dirname(os.path.dirname(SRC)))
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(root, "csrc", "include"), "-I" + cuda, str(prog), "-o", str(tmp_path / "level")], check=True)
    env = {k: v for k, v in os.environ.items() if k != "BLAZE_PDL"}
    got = [subprocess.run([str(tmp_path / "level")], env={**env, **e}, capture_output=True, text=True).stdout for e in ({}, {"BLAZE_PDL": "0"}, {"BLAZE_PDL": "1"})]
    assert got == ["1 0", "0 0", "1 1"]
    folder = os.path.dirname(SRC)
    for f in sorted(os.listdir(folder)):
        text = open(os.path.join(folder, f)).read()
        for at in re.finditer("cudaLaunchAttributeProgrammaticStreamSerialization", text):
            near = text[max(0, at.start() - 600):at.start() + 1500]
            assert "pdl_enabled()" in near or "pdl_pairs()" in near, f


def test_kernel_attributes_are_set_for_every_device():
    """A limit of shared memory that is set for the process's first device only does not hold on its second."""
    folder = os.path.dirname(SRC)
    host = open(os.path.join(os.path.dirname(folder), "include", "blaze", "host.h")).read()
    once = host[host.index("struct PerDeviceOnce"):]
    assert host.count("cudaFuncSetAttribute(") == 1 and once.index("done[dev]") < once.index("cudaFuncSetAttribute(") < once.index("\n};")
    for f in sorted(os.listdir(folder)):
        assert "cudaFuncSetAttribute(" not in open(os.path.join(folder, f)).read(), f
