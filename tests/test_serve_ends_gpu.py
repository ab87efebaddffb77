"""A serving call that raises in the middle: nothing it launched writes to the
server's memory afterwards."""
import dataclasses

import pytest
import torch

from pageflow_b200 import serve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("after_s", [0.0, 0.002, 0.004])
def test_no_launch_outlives_a_call_that_raises(after_s):
    dev = torch.device("cuda", 0)
    n = 200_000_000
    spec = dataclasses.replace(serve.scaled(serve.SERVE, 1000), fact_rows=n, probe_min=n, probe_max=n)
    server = serve.Server(serve.Dimensions(spec, dev), serve.FactPool(spec, dev),
                          n * 20 + (1 << 30), dev, pinned_bytes=1 << 26)
    requests = serve.make_requests(spec, 40, seed=1)   # 8 billion rows: tens of milliseconds
    with pytest.raises(TimeoutError):
        server.run(requests, timeout_s=after_s)
    assert server.stream.query() and server.copy_stream.query()
