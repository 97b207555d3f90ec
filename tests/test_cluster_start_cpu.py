"""Distributed shared memory: a CTA's shared memory may be accessed from its cluster once that CTA has started, which only a
cluster barrier shows.  In every kernel of the library that addresses a peer's shared memory, a cluster barrier's wait stands
before the first such address."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "dmrg_b200", "csrc")
REMOTE = re.compile(r"map_shared_rank\(|mapa\.shared::cluster|leader_addr\(|umma_commit_pair\(")
WAIT = re.compile(r"barrier\.cluster\.wait|cluster\.sync\(\)|pair_sync\(\)")


def _kernels(text):
    """(name, body) of the __global__ functions of a source file."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        i = text.index("{", m.end())
        name = re.findall(r"(\w+)\s*\(", text[m.end() : i].replace("__launch_bounds__", ""))
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield next(n for n in reversed(name) if n.endswith("kernel") or "_" in n), text[i:j]


def test_cluster_barrier_before_the_first_remote_address():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            for name, body in _kernels(f.read()):
                first = REMOTE.search(body)
                if first:
                    found.append(name)
                    wait = WAIT.search(body)
                    assert wait and wait.start() < first.start(), f"{os.path.basename(path)}: {name}"
    assert {"jacobi_round_kernel", "qr_panel_kernel", "orth_one_kernel", "matvec_fused_kernel", "gemm_f64_kernel", "gemm_i8_pair_kernel"} <= set(found), found
