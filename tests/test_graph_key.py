"""A captured evaluation is replayed only for plans whose tables lie where it reads them:
every offset that the captured launches use is part of the graph's key."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "hawkes_b200", "csrc", "hphc_executor.cpp")


def test_every_table_offset_is_in_the_key():
    text = open(SRC).read()
    launches = text[text.index("int Executor::launch_sequence(int grid) {"):]
    launches = launches[:launches.index("\n}\n")]
    used = set(re.findall(r"\boff\w+_\b", launches))
    assert len(used) >= 6
    key = re.search(r"const size_t offsets\[\] = \{([^}]*)\};", text)
    assert key and used <= set(re.findall(r"\boff\w+_\b", key.group(1)))
    assert re.search(r"key == last", text)
