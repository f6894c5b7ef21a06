"""A mesh with two edges between the same vertices is turned down by the member-row tables: both would add
their term to one slot of the edge pass at the same time."""
import numpy as np

from test_rows import lib, run  # noqa: F401


def theta():
    """Three cells around two vertices, joined by three edges."""
    m = dict(nCells=3, nEdges=3, nVertices=2, maxEdges=2, maxEdges2=4)
    m['cellsOnEdge'] = np.array([[1, 3], [1, 2], [2, 3]])
    m['verticesOnEdge'] = np.array([[1, 2]] * 3)
    m['edgesOnEdge'] = np.array([[2, 3, 0, 0], [1, 3, 0, 0], [2, 1, 0, 0]])
    m['nEdgesOnEdge'] = np.array([2, 2, 2])
    m['edgesOnCell'] = np.array([[1, 2], [2, 3], [3, 1]])
    m['nEdgesOnCell'] = np.array([2, 2, 2])
    m['cellsOnVertex'] = np.array([[1, 2, 3]] * 2)
    m['edgesOnVertex'] = np.array([[1, 2, 3]] * 2)
    for n, s in (('weightsOnEdge', (3, 4)), ('kiteAreasOnVertex', (2, 3)), ('dcEdge', 3), ('dvEdge', 3), ('areaCell', 3),
                 ('areaTriangle', 2)):
        m[n] = np.ones(s)
    for p, n in (('Cell', 3), ('Edge', 3), ('Vertex', 2)):
        for x in 'xyz':
            m[x + p] = np.linspace(0.1, 1.0, n) * (1 + 'xyz'.index(x))
    return m


def test_parallel_edges_are_turned_down(lib):  # noqa: F811
    rc, err, _ = run(lib, theta(), 0)
    assert rc == 1 and 'same vertices' in err
