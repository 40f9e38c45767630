"""The stream pool of the file pipelines: an idle stream goes to one caller,
on its own device, and no more than LIMIT are kept."""
from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from mojoalign_b200 import streams  # noqa: E402


@pytest.mark.parametrize("extra", [0, 1, 5])
def test_idle_streams_are_bounded_and_given_once(monkeypatch, extra):
    monkeypatch.setattr(streams, "_FREE", {})
    made = []

    def make(device):
        made.append(SimpleNamespace(device=device))
        return made[-1]

    monkeypatch.setattr(torch.cuda, "Stream", lambda device: make(device))
    held = [streams.take("cuda:1") for _ in range(streams.LIMIT + extra)]
    assert len({id(s) for s in held}) == len(held)
    for s in held:
        streams.give(s)
    assert streams.take("cuda:0") is made[-1] and made[-1] not in held  # another device's are not handed out
    n = len(made)
    with ThreadPoolExecutor(8) as pool:
        again = list(pool.map(lambda _: streams.take("cuda:1"), range(streams.LIMIT)))
    assert len(made) == n and len({id(s) for s in again}) == streams.LIMIT
    assert all(any(s is h for h in held) for s in again)
