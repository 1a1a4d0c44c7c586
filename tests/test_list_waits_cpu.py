"""The waits of the list launch that lie behind one another: who waits for a waiter waits longer.  Read from the sources, since a wait that is
given up too early shows only where a CTA is held up for seconds."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "p40-kernel_b200", "csrc", "gemv_chain.cuh")).read()


def function(head):
    body = SOURCE[SOURCE.index(head):]
    return body[:body.index("\n}")]


def test_an_image_is_waited_for_longer_than_its_writer_waits():
    """A part of an image is written behind a wait for the rows of other CTAs; both waits are counted in trips to L2 with sleeps of some 32 to
    64 ns.  At 0.6 us and more per trip a quarter more trips are longer whatever the sleeps take."""
    value = lambda text: eval(text.replace("u", ""), {})
    polls = {name: value(v) for name, v in re.findall(r"\b(CHAIN_\w+_POLLS) = ([^,;]+)", SOURCE)}
    writer = re.search(r"n < \(?([^;)]+)\)?;", function("bool grid_counter_wait("))[1]
    assert 4 * polls["CHAIN_IMAGE_POLLS"] >= 5 * (polls[writer] if writer in polls else value(writer))
