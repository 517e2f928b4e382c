"""One NeighborQuery queried by several threads at once, each with radii and neighbour numbers of its
own, more of them than the object keeps grids for (four): the lists and counts of one thread alone."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ask(freud, nq, queries, what):
    kind, value = what
    if kind == "rdf":
        rdf = freud.density.RDF(30, value)
        rdf.compute(nq, query_points=queries, neighbors=dict(r_max=value, exclude_ii=False))
        return [np.array(rdf.bin_counts_u64)]
    q = queries if kind.endswith("other") else np.asarray(nq.points)
    args = dict(num_neighbors=value) if kind.startswith("knn") else dict(r_max=value)
    nl = nq.query(q, dict(args, exclude_ii=not kind.endswith("other"))).toNeighborList(
        sort_by_distance=kind == "sorted")
    return [np.array(nl[:]), np.array(nl.distances)]


@pytest.mark.parametrize("structure", ["linkcell", "aabb", "cellquery"])
def test_threads(freud, structure):
    rs = np.random.RandomState(4)
    L = 28.0
    box = freud.box.Box.cube(L)
    pts = ((rs.random_sample((22000, 3)) - 0.5) * L).astype(np.float32)
    queries = ((rs.random_sample((9000, 3)) - 0.5) * L).astype(np.float32)
    make = {"linkcell": lambda: freud.locality.LinkCell(box, pts, 1.0), "aabb": lambda: freud.locality.AABBQuery(box, pts),
            "cellquery": lambda: freud.locality.CellQuery(box, pts)}[structure]
    # radii of groups, of their half (the same cells, by index), of the block kernels; one list and the next of
    # a thread ask for different grids
    work = [[("own", 1.0), ("own", 2.0), ("sorted", 1.0), ("other", 1.6)],
            [("sorted", 2.0), ("own", 1.0), ("rdf", 1.0), ("own", 2.6)],
            [("other", 1.3), ("rdf", 2.0), ("own", 0.8), ("sorted", 0.5)]]
    if structure != "cellquery":
        work.append([("knn", 6), ("own", 1.8), ("knn other", 12), ("knn", 40)])
    want = [[ask(freud, make(), queries, w) for w in one] for one in work]
    nq = make()
    errors = []

    def run(one, expected):
        try:
            for _ in range(12):
                for w, e in zip(one, expected):
                    for a, b in zip(ask(freud, nq, queries, w), e):
                        np.testing.assert_array_equal(a, b)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=x) for x in zip(work, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
