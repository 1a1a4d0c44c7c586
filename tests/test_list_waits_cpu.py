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


def image_poll():
    loop = SOURCE[SOURCE.index("image_load2(table_image"):]
    return loop[:loop.index("__nanosleep(")]


def test_a_warp_leaves_the_poll_of_an_image_as_a_whole():
    """The poll votes with all 32 lanes, and what one lane reads of another warp's word may not be what its neighbour reads."""
    exits = [line for line in image_poll().splitlines() if "break;" in line]
    assert len(exits) >= 2
    for line in exits:
        alone = re.sub(r"__(all|any)_sync\(0xffffffffu, [^()]*\)", "", line.split("//")[0])
        assert "there" not in alone and "stop" not in alone, line


def test_a_poll_that_ends_for_another_warp_reports_nothing():
    """A warp that was told to leave (*stop) does not write over what the one that gave up has put into the status word."""
    after = SOURCE[SOURCE.index("image_load2(table_image"):]
    report = next(line for line in after.splitlines() if "STATUS_GRID_TIMEOUT" in line)
    assert re.search(r"if \(lane == 0 && !\*stop\)", report), report
