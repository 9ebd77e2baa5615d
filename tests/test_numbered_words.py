"""The exchange words of the resident sweeps are a value and the number of the
half sweep it belongs to, 8 bytes. Whoever polls them takes the value on the
number's word, so both have to be one access: the accesses' element width is the
word's on either side."""
import os
import re

HERE = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_words_are_read_as_they_are_written():
    with open(os.path.join(HERE, "vapor_b200", "csrc", "sor_resident.cuh")) as f:
        source = f.read()
    stores = re.findall(r"\bst\.relaxed\.(?:gpu|cluster)[\w.:]*", source)
    loads = re.findall(r"\bld\.(?:volatile|relaxed|acquire)[\w.:]*", source)
    assert stores and loads
    assert all(op.endswith(".v2.b64") for op in stores + loads), loads
    assert all(op.startswith(("ld.relaxed.gpu.global", "ld.relaxed.cluster.shared::cta")) for op in loads), loads
