"""The bench's kernel labels, without a GPU: the commit workload's roofline names the kernel that its
transforms run, and reads that kernel's captured traffic at the workload's own size."""
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_commit_roofline_names_the_kernel_it_times():
    import bench
    with open(os.path.join(ROOT, "binius64_b200", "csrc", "ntt.cu")) as f:
        src = f.read()
    assert re.search(r"__global__ void[^;{]*\b%s\(" % bench.COMMIT_KERNEL, src)
    # the sizes for which the transforms leave the tensor-core passes (tc_tile_bits)
    rule = re.search(r"if \(log_d < (\d+) && log_d - skip_early <= kTcMinTileBits\) return 0;", src)
    assert bench.LOG_LEN + bench.LOG_BATCH >= int(rule.group(1))
    assert bench.COMMIT_KERNEL == "ntt_tc_pass_kernel"
    name = f"{bench.COMMIT_KERNEL}_log{bench.LOG_LEN}_b{bench.LOG_BATCH}.md"
    with open(os.path.join(ROOT, "profiles", name)) as f:
        assert bench.COMMIT_KERNEL in f.readline()
    traffic = bench.profiled_traffic(name)
    elems = 1 << (bench.LOG_LEN + bench.LOG_BATCH)
    # a pass reads and writes the codeword once; what stays in the L2 is not written back
    assert 0.8 * 32 * elems <= traffic <= 1.05 * 32 * elems
