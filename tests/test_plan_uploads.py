"""A plan's device arrays, read from the source: each one that is uploaded is
read by a launch, released and counted."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpir_b200", "csrc")


def test_uploaded_arrays_are_used():
    text = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            text[os.path.basename(path)] = f.read()
    whole, factor = "".join(text.values()), text["factor.cu"]
    up = factor[factor.index("void Plan::upload_all("):factor.index("void Plan::release_device(")]
    names = re.findall(r"^\s*(\w+)\s*=\s*upload\((\S+), s\);", up, re.M)
    assert len(names) > 20
    sizes = factor[factor.index("size_t Plan::upload_bytes("):factor.index("void Plan::upload_all(")]
    for name, host in names:
        assert re.search(rf"\b{name}\.as<", whole), f"{name}: no kernel reads it"
        assert len(re.findall(rf"&{name}\b", factor)) == 2, f"{name}: release_device and device_bytes"
        assert f"b({host})" in sizes, f"{host}: upload_bytes"
