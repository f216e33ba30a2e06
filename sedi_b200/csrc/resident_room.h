// Room on the GPU for the resident solvers' launches (host arithmetic only).
//
// The blocks of a grouped launch wait for one another, so all of them must
// find room: two such launches that each hold a part of the GPU and wait for
// the rest would wait until their limit.  Launches of single-block groups end
// by themselves, but may hold every SM for a whole batch, longer than that
// limit.  A new launch therefore waits (on its stream) for the oldest ones
// until those it may overlap and itself have room, where one of them is
// grouped; single-block launches alone need none.  Other kernels are short.
//
// A launch is charged the SMs it may touch, a block each: nothing makes the
// scheduler put two blocks on an SM that has room for them (256 blocks of
// 64^3 x 8 lanes, two an SM, charged 128 SMs would leave 20 to another launch
// that all 148 are taken from).
#pragma once

#include <cstddef>
#include <vector>

namespace sedi {

struct RoomUse {
	int held = 0;          // SMs the launch may touch
	bool grouped = false;  // its blocks wait for one another
};

inline RoomUse room_use(int blocks, int group, int sms) {
	RoomUse u;
	u.held = blocks < sms ? blocks : sms;
	u.grouped = group > 1;
	return u;
}

// Which of the launches that may still be running (oldest first) one of `u`
// has to wait for.
inline std::vector<char> room_waits(const std::vector<RoomUse> &running, const RoomUse &u, int sms) {
	std::vector<char> wait(running.size(), 0);
	long total = u.held, groups = u.grouped;
	for (const RoomUse &r : running) {
		total += r.held;
		groups += r.grouped;
	}
	for (size_t i = 0; i < running.size() && total > sms && groups > 0; i++) {
		if (!u.grouped && !running[i].grouped) continue;
		wait[i] = 1;
		total -= running[i].held;
		groups -= running[i].grouped;
	}
	return wait;
}

}  // namespace sedi
