"""Clears and copies of a world's device memory go through its own stream: on the legacy default stream
nothing orders them with the kernels, whose streams do not wait for it (cudaStreamNonBlocking)."""
import os
import re

import pytest

from jbgpu._build import CSRC

# everything that works on a world's stream (the network of mlp.cu has a stream of its own)
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and not f.startswith("mlp"))


@pytest.mark.parametrize("name", FILES)
def test_no_clear_or_copy_on_the_default_stream(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert not re.findall(r"\bcuda(?:Memset|Memcpy)(?:2D)?\(", text)
    for call in re.findall(r"\bcudaMem(?:set|cpy)Async\(([^;]*?)\)(?:\)|;| !=| \|\|| ==)", text):
        last = call.rsplit(",", 1)[-1].strip()
        assert last in ("s", "a", "w->stream", "stream"), call
