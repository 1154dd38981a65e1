"""Every stage reports what it finds wrong in a status word, the ordering of the output among them (a key
that names no row, a look-back that gives up: conditions that no input brings about).  On the CPU: a join
reads that word back after its last stage, whatever its options."""
import re
from pathlib import Path

API = Path(__file__).resolve().parents[1] / "tensorjoin_variants_b200" / "csrc" / "tj_api.cu"


def test_status_is_read_after_the_ordering():
    text = re.sub(r"//[^\n]*", "", API.read_text())
    body = text[text.index("void run_batch_body("):text.index("void run_batch(")]
    ordered = max(body.index("order_rows("), body.rindex("radix_sort("), body.index("rows_batch_offsets("))
    read = re.compile(r"TJ_CUDA\(cudaMemcpyAsync\(&(\w+), &ctr\.p->status, 8, cudaMemcpyDeviceToHost, st\)\);"
                      r"\s*TJ_CUDA\(cudaStreamSynchronize\(st\)\);\s*check_status\(\1\);").search(body, ordered)
    assert read, "the status word is not read after the last stage"
    before = body[:read.start()].rstrip()
    assert before[-1] in ";}", "the read depends on a condition"
    assert before.count("{") - before.count("}") == 1, "the read lies inside a block"
