"""A CTA's shared memory may be written by the other CTAs of its cluster only once
it has started (CUDA programming guide, distributed shared memory).  Whether a
kernel keeps to that does not show in its results, except when a CTA starts late,
so it is read from the source: between its entry and the first exchange, the
cluster form of the resident CG passes a barrier of the whole cluster."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ufc-fem-kernel_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_only_the_resident_cg_writes_across_ctas():
    users = [f for f in sorted(os.listdir(CSRC))
             if f.endswith((".cu", ".cuh")) and re.search(r"map_shared_rank|\bmapa\b|shared::cluster\.global", _code(f))]
    # (block.cu's bulk copies name the cluster window for their own CTA: no cluster launch there)
    assert users == ["block.cu", "resident.cu"]
    assert "map_shared_rank" not in _code("block.cu") and "ClusterDimension" not in _code("block.cu")


def test_cluster_barrier_before_the_first_exchange():
    text = _code("resident.cu")
    body = text[text.index("k_cg_resident(const ResArgs A) {"):]
    body = body[:body.index("\n}\n")]
    lam = re.search(r"auto reduce = .*?\n  \};\n", body, flags=re.S)
    assert "map_shared_rank" in lam.group(0)
    body = body[:lam.start()] + body[lam.end():]  # the exchange itself; its calls stay
    assert "map_shared_rank" not in body
    before = body[:body.index("reduce(")]
    assert re.search(r"if constexpr \(SYNC == kCluster\)\s*cg::this_cluster\(\)\.sync\(\);", before)
