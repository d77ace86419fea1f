"""Products of one accumulator and shape follow each other on the tensor core; between others only a commit says that one is done.  Where a
product overwrites tensor memory that another reads as its operand, the thread that issues it waits for that one's commit.  (A race is not
something a test can wait for: the source is read.)"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kfold_b200", "csrc")


def test_transition_scores_wait_for_the_product_that_reads_the_hidden_channels():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "transition_pair.cu")).read())
    scores = text.index("mma_f16_ss_pair(d")                    # S, over the h of the chunk that had its buffer
    waits = re.findall(r"mbar_wait\(&(\w+)\[s1\]", text[:scores])
    assert len(waits) == 1
    reader = text.index("mma_f16_ts_pair(")                     # O, which reads that h
    after = text[reader:text.index("++s2", reader)]
    assert f"tc_commit_pair(&{waits[0]}[s2])" in after
    assert not re.search(r"mbar_arrive\w*\(&" + waits[0], text)
