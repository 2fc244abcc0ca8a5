"""Under which name the benchmark's tables count a kernel (the designs' tables ask for an operation by one name)."""
import re
from pathlib import Path

import bench

CSRC = Path(bench.__file__).parent / "longbow-quarrel_b200" / "csrc"


def test_forms_of_one_operation_count_under_its_name():
    assert bench._kind("void (anonymous namespace)::chunk_out_kernel<64, 64, 0, true>(ChunkArgs)") == ("linear_scan", 1)
    assert bench._kind("chunk_state_kernel<64>") == ("linear_scan", 0) and bench._kind("linear_scan_kernel<float>") == ("linear_scan", 1)
    assert bench._kind("moe_up_rows_kernel<4, 2, true>") == ("moe_up", 1) and bench._kind("latent_prefill_kernel") == ("latent_attention_tc", 1)
    assert bench._kind("gemm_tc_kernel<256>") == ("gemm_tc", 1) and bench._kind("x" * 50) == ("x" * 40, 1)


def test_every_renamed_kernel_is_one_that_the_sources_have():
    kernels = set(re.findall(r"\b(\w+)_kernel\(", "".join(p.read_text() for p in CSRC.glob("*.cu"))))
    assert set(bench._COUNTED_AS) <= kernels
