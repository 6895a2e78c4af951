"""Requests that cannot be served, and a launch that fails, on the host: streams, uploads and
launches are fakes. A bad request is refused before anything is launched for another one, and
after any error no stream has work left and the server's room and slots are as they were."""

import contextlib
import dataclasses

import numpy as np
import pytest
import torch

from nabladyn_b200.serving import ReplicaRequest, _server


class Stream:
    def __init__(self, *args, **kwargs):
        self.waits = 0

    def synchronize(self):
        self.waits += 1


@pytest.fixture
def server(monkeypatch):
    streams = []

    def stream(*args, **kwargs):
        streams.append(Stream())
        return streams[-1]

    monkeypatch.setattr(torch.cuda, "Stream", stream)
    monkeypatch.setattr(torch.cuda, "current_stream", stream)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    made = object.__new__(_server.ReplicaServer)
    made.device, made.max_slots, made.capacity = torch.device("cpu"), 8, 1 << 16
    made.round_atom_steps, made.stage_ahead = 10_000, 4
    made.large_atoms, made.large_round_steps = 1000, 50
    made._free_units = [(0, made.capacity // _server._ALIGN)]
    made._free_slots = list(range(8))
    made.streams, made.calls = streams, []
    monkeypatch.setattr(made, "_place", lambda *a: made.calls.append("place"), raising=False)
    monkeypatch.setattr(made, "_launch", lambda *a: made.calls.append("launch"), raising=False)
    monkeypatch.setattr(made, "_team", lambda *a: 1, raising=False)
    return made


def request(n, **changes):
    given = ReplicaRequest(positions=np.zeros((n, 3)), velocities=np.zeros((n, 3)),
                           masses=np.full(n, 39.948), cell=np.full(3, 5.0), temperature=90.0,
                           steps=10, name=n)
    return dataclasses.replace(given, **changes)


@pytest.mark.parametrize("bad, error", [
    ({"cell": np.array([5.0, 5.0, 1.5])}, ValueError),   # below twice the cutoff
    ({"cell": np.array([5.0, np.inf, 5.0])}, ValueError),
    ({"masses": np.float64(39.948)}, IndexError),
    ({"masses": np.full(63, 39.948)}, ValueError),
    ({"velocities": np.zeros((63, 3))}, ValueError),
    ({"velocities": np.zeros((64, 2))}, ValueError),
    ({"positions": np.zeros((64, 2))}, ValueError),
    ({"velocities": [["a", "b", "c"]] * 64}, ValueError),
])
@pytest.mark.parametrize("arrival", [0.0, 3600.0])
def test_a_bad_request_is_refused_before_any_launch(server, bad, error, arrival):
    free = list(server._free_units), list(server._free_slots)
    with pytest.raises(error):
        server.serve([request(2000), request(64, arrival=arrival, **bad)])
    assert server.calls == []
    assert (server._free_units, server._free_slots) == free


def test_what_an_admission_takes_is_accepted(server):
    for given in ({"masses": np.full(1, 39.948)}, {"velocities": np.zeros(3)},
                  {"velocities": np.zeros((1, 64, 3), dtype=np.float32)},
                  {"positions": torch.zeros(64, 3)}, {"masses": [39] * 64}):
        server._check(request(64, **given))
        assert server._stage(request(64, **given)).record.num_atoms == 64


def test_a_failed_launch_leaves_nothing_running_and_nothing_taken(server, monkeypatch):
    free = list(server._free_units), list(server._free_slots)

    def launch(slots, budgets, mode, lane="", team=1):
        server.calls.append(lane)
        if lane == "":  # the small replicas', behind the large ones'
            raise RuntimeError("launch failed")

    monkeypatch.setattr(server, "_launch", launch, raising=False)
    monkeypatch.setattr(server, "_table_copy", lambda lane: (None, None), raising=False)
    with pytest.raises(RuntimeError, match="launch failed"):
        server.serve([request(2000), request(64)], realtime=False)
    assert "_large" in server.calls
    assert all(stream.waits for stream in server.streams[-3:])
    assert (server._free_units, server._free_slots) == free
