"""The barrier protocol of the CTA pairs of the 4-bit tensor GEMM
(parpar_gb300/csrc/k_tc4.cu: k_tc4_gemm), checked on the CPU.

The source test holds every signal between the two CTAs of a pair to cluster
scope: an arrival or a wait at CTA scope orders nothing between them."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parpar_gb300", "csrc", "k_tc4.cu")

# who gives a barrier's signals: its own CTA alone, either CTA (or MMAs that
# read the shared memory of both), or accumulators changing hands
OWN = {"QFULL", "QEMPTY", "BFULL"}
PAIR = {"READY", "EMPTY", "IDFULL", "IDEMPTY"}
TMEM = {"TFULL", "TEMPTY"}


def source():
    with open(SRC) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    # adjacent string literals are one string
    return re.sub(r'"\s*\n\s*"', "", text)


def test_signals_between_the_ctas_of_a_pair_have_cluster_scope():
    text = source()
    # arrivals that can reach the other CTA
    arrivals = re.findall(r"[^\"]*mbarrier\.arrive[a-z_:.]*shared::cluster\.b64 _[^\"]*", text)
    assert arrivals
    for a in arrivals:
        assert "mbarrier.arrive.release.cluster." in a or (
            "fence.release.sync_restrict::shared::cta.cluster;" in a and "mbarrier.arrive.relaxed.cluster." in a), a
    # waits, by the barrier they wait for
    waits = re.findall(r"t4_wait_ab(<[^>]*>)?\([^;]*?T4B_([A-Z]+)", text)
    assert {b for _, b in waits} == OWN | PAIR | TMEM
    for kind, b in waits:
        assert kind == ("" if b in OWN else "<T4_PAIR>" if b in PAIR else "<T4_TMEM>"), (kind, b)
    body = text[text.index("bool t4_try("):text.index("uint32_t t4_test_pair(")]
    near, far = body[body.index("if(BY != T4_CTA)"):].split("else", 1)
    assert "try_wait.parity.relaxed.cluster." in near and "try_wait.parity.shared::cta" in far
    body = text[text.index("bool t4_wait_ab("):]
    assert re.search(r"if\(t4_try<BY>\(bar, parity\)\) \{\s*if\(BY == T4_PAIR\) t4_acquire_pair\(\);\s*return true;", body)
    assert "fence.acquire.sync_restrict::shared::cluster.cluster;" in text
    # a stage found ready by the look ahead is acquired where its wait is skipped
    assert re.search(r"if\(seen\) t4_acquire_pair\(\);\s*else if\(.*T4B_READY", text)
    assert "test_wait.parity.relaxed.cluster." in text
    # the accumulators' signals stand between the tcgen05 fences
    for b in TMEM:
        m = re.search(r"t4_wait_ab<T4_TMEM>\([^;]*T4B_%s[^;]*;\s*(break; \}|)\s*([^;]*;)" % b, text)
        assert m and "tcgen05.fence::after_thread_sync" in m.group(2), (b, m)
