"""What planning a model touches: a weight that is folded, merged and joined is not copied on the way."""
import resource

from fluidml_b200 import models
from fluidml_b200.executor import Executor


def pages_touched(data, precision):
    before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
    Executor.make_plain_greedy("t").set_option("gemm_precision", precision).plan(data)
    return resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before


def test_joining_products_copies_no_weights():
    data = models.build_gpt_neox(layers=4, hidden=768, heads=12, ffn=3072, vocab=100, batch=1, seq=40).to_bytes()
    pages_touched(data, "3xtf32")                                      # lazily loaded code, the allocator's first pages
    apart, joined = pages_touched(data, "3xtf32"), pages_touched(data, "auto")
    assert joined - apart < 0.1 * len(data) / resource.getpagesize()   # one copy of the weights is all of it
