"""Region and its subclasses copy and pickle as what they are, whether or not
the C struct of the region has been built."""
import copy
import pickle
from dataclasses import dataclass

import itkg


@dataclass(frozen=True)
class Named(itkg.Region):
    name: str = ""


def test_copies():
    for r in (itkg.Region((1, -2), (3, 4)), Named((0, 0, 5), (6, 7, 8), "roi")):
        for built in (False, True):
            if built:
                assert tuple(r._c().size)[:r.dim] == r.size
            for other in (copy.copy(r), copy.deepcopy(r), pickle.loads(pickle.dumps(r))):
                assert type(other) is type(r) and other == r and hash(other) == hash(r)
                assert tuple(other._c().index)[:r.dim] == r.index
