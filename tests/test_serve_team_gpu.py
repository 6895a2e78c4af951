"""Replicas advanced by a cluster of CTAs: every team size gives the same bits as one CTA, on the
cell grid and on the all-pairs path, at the sizes where the rows divide unevenly among the CTAs
(just around two CTAs' worth of atoms, a last CTA with a single row, eight CTAs), through
rebuilds and in several rounds. The sums over a replica's rows are taken in one order whatever
the team, so nothing is left to a tolerance."""

import numpy as np
import pytest

from nabladyn_b200.serving import ReplicaRequest, ReplicaServer, _server

pytestmark = pytest.mark.gpu

A = 0.5745  # fcc lattice constant (nm)
SITES = np.array([[0, 0, 0], [0, 1, 1], [1, 0, 1], [1, 1, 0]]) / 2


def lattice_request(cells, atoms, steps, seed):
    rng = np.random.default_rng(seed)
    grid = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1)
    positions = ((grid.reshape(-1, 1, 3) + SITES).reshape(-1, 3) * A)
    positions = positions[np.sort(rng.permutation(len(positions))[:atoms])]
    positions = positions + rng.normal(0.0, 0.01, positions.shape)
    return ReplicaRequest(positions=positions, velocities=rng.normal(0.0, 0.3, positions.shape),
                          masses=np.full(atoms, 39.948), cell=np.array(cells) * A,
                          temperature=300.0, steps=steps, name=f"{atoms}")


@pytest.mark.parametrize("cells, atoms", [
    ((9, 9, 9), 2047), ((9, 9, 9), 2048), ((9, 9, 9), 2561), ((13, 13, 13), 8193),
    ((13, 13, 13), 8788), ((16, 16, 4), 4096)])
def test_every_team_gives_the_same_bits(cuda, monkeypatch, cells, atoms):
    request = lattice_request(cells, atoms, 60, seed=atoms)
    results = []
    for team in (1, 2, 4, 8):
        monkeypatch.setattr(ReplicaServer, "_team", lambda self, active, work, team=team: team)
        server = ReplicaServer(device=cuda, budget_bytes=64 << 20, max_slots=2,
                               round_atom_steps=25 * atoms)
        results.append(server.serve([request], realtime=False)[0])
    one = results[0]
    assert one.status == 0 and one.steps == 60 and one.rebuilds >= 2
    for other in results[1:]:
        np.testing.assert_array_equal(other.positions, one.positions)
        np.testing.assert_array_equal(other.velocities, one.velocities)
        np.testing.assert_array_equal(other.images, one.images)
        assert (other.energy, other.rebuilds, other.status) == (one.energy, one.rebuilds, 0)


@pytest.mark.parametrize("team", (1, 2, 8))
def test_a_room_that_begins_at_an_odd_atom(cuda, monkeypatch, team):
    """The per-32-row sums of a team lie in per-atom memory: a replica whose room begins at atom
    33 (and one of 33,000 atoms, whose sums a single CTA keeps there as well) gives the bits it
    gives at atom 0."""
    monkeypatch.setattr(ReplicaServer, "_team", lambda self, active, work: team)
    atoms = 33000 if team == 1 else 4000
    first = lattice_request((5, 5, 5), 20, 3, seed=1)
    request = lattice_request((21, 21, 21) if team == 1 else (10, 10, 10), atoms, 12, seed=2)
    alone = ReplicaServer(device=cuda, budget_bytes=64 << 20, max_slots=2)
    expected = alone.serve([request], realtime=False)[0]
    monkeypatch.setattr(_server, "_ALIGN", 33)
    server = ReplicaServer(device=cuda, budget_bytes=64 << 20, max_slots=2, large_atoms=None)
    results = {r.num_atoms: r for r in server.serve([first, request], realtime=False)}
    got = results[atoms]
    assert got.status == expected.status == 0 and got.steps == 12
    np.testing.assert_array_equal(got.positions, expected.positions)
    np.testing.assert_array_equal(got.velocities, expected.velocities)
    assert got.energy == expected.energy
