"""Which forwards of an engine are replayed from a CUDA graph."""
from __future__ import annotations

from collections import OrderedDict


class Graphs:
    """At most ``limit`` graphs, by a key that determines the launches.

    A key's first forward runs as plain launches and its second one is captured while there is room.  When there is none, a
    graph gives way only after ``idle`` forwards without a use, the one unused for longest first; until then the other keys stay
    on plain launches.  A capture costs several forwards, and with more keys in turn than graphs every capture would throw out a
    graph that is about to be used: at most ``limit`` captures per ``idle`` forwards are left.  The last ``keys`` keys are known.

    Measured on a B200, us a call with every call waited for, first in first out before -> this rule: queries of 5 to 60 tokens
    over 16 graphs 1418 -> 1126 (of 5 to 15 tokens, where all fit, 912 both), 1 to 64 images of ViT-B/16 over 8 graphs
    2510 -> 1749 (1 to 8 images, three sizes: 1010 both)."""

    def __init__(self, limit: int, keys: int = 256, idle: int = 256):
        self.limit, self.keys, self.idle = limit, keys, idle
        self.seen: OrderedDict = OrderedDict()       # keys of earlier forwards without a graph, the one unused for longest first
        self.graphs: OrderedDict = OrderedDict()     # key -> [graph, forward of its last use], likewise
        self.clock = 0

    def use(self, key):
        """A forward of ``key`` begins.  ``(new, graph, capture)``: whether ``key`` is unknown, its graph if it has one, and
        whether the caller is to capture one now and hand it to ``put``."""
        self.clock += 1
        entry = self.graphs.get(key)
        if entry is not None:
            entry[1] = self.clock
            self.graphs.move_to_end(key)
            return False, entry[0], False
        new = key not in self.seen
        self._remember(key)
        if new or self.limit < 1:
            return new, None, False
        if len(self.graphs) >= self.limit:
            oldest, (_, last) = next(iter(self.graphs.items()))
            if self.clock - last < self.idle:
                return new, None, False
            self.graphs.pop(oldest)
            self._remember(oldest)
        return new, None, True

    def put(self, key, graph) -> None:
        self.graphs[key] = [graph, self.clock]
        self.seen.pop(key, None)

    def _remember(self, key) -> None:
        self.seen[key] = True
        self.seen.move_to_end(key)
        if len(self.seen) > self.keys:
            self.seen.popitem(last=False)
