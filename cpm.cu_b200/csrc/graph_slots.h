// Which decode passes are captured as graphs.  A pass of a shape (2 * tokens + (tree mask given): at most 128 of them) is captured
// the second time it comes, while a slot is free.  After that a graph gives its slot up only when none of the last kPatience passes
// replayed it, so that a caller whose trees go through more shapes than there are slots pays for a capture once in a while
// at most (16 per 256 passes; a capture and its instantiation cost as much as a few passes) and the shapes without a slot
// run launch by launch.
#pragma once
#include <map>

class GraphSlots {
public:
    enum Act { PLAIN = 0, CAPTURE = 1, REPLAY = 2 };
    static constexpr int kSlots = 16, kPatience = 256;

    // What the next pass, of shape `key`, does; with CAPTURE `evict` is the shape whose graph goes first, or -1.
    Act pass(int key, int& evict) {
        evict = -1;
        ++now_;
        Shape& s = shapes_[key];
        if (s.held) {
            s.last = now_;
            return REPLAY;
        }
        if (s.barred || s.passes++ == 0) return PLAIN;
        if (held_ >= kSlots) {
            auto oldest = shapes_.end();
            for (auto it = shapes_.begin(); it != shapes_.end(); ++it) {
                if (it->second.held && (oldest == shapes_.end() || it->second.last < oldest->second.last)) oldest = it;
            }
            if (now_ - oldest->second.last <= kPatience) return PLAIN;
            oldest->second.held = false;
            --held_;
            evict = oldest->first;
        }
        s.held = true;
        s.last = now_;
        ++held_;
        return CAPTURE;
    }

    // The capture of `key` did not succeed: its passes run launch by launch from now on.
    void bar(int key) {
        Shape& s = shapes_[key];
        if (s.held) --held_;
        s.held = false;
        s.barred = true;
    }

private:
    struct Shape {
        long passes = 0, last = 0;
        bool held = false, barred = false;
    };
    std::map<int, Shape> shapes_;
    long now_ = 0;
    int held_ = 0;
};
