// once.hpp -- tables that are built on first use.
#pragma once

// make() until it has succeeded once (0): `built` is set after it only, so that a
// build which failed half way (an allocation, a launch) is made anew by the next
// call instead of being taken for done.
template <class Make>
auto build_once(bool& built, Make&& make) -> decltype(make()) {
  if (built) return decltype(make()){};
  const auto s = make();
  if (!s) built = true;
  return s;
}
